"""GPT decoder (lua/luatorch/models/gpt.lua).

`GPT(vocab_size, embed_dim, num_heads, num_layers, max_seq_len, dropout=0.1)`: token
embedding + positional encoding + embedding dropout + N pre-LN transformer blocks + final
LayerNorm + UNTIED head Linear(embed, vocab, bias=False).  `forward(input[B, S])` returns
logits [B*S, vocab]; `generate(prompt, max_tokens, temperature, top_k)` samples token by token,
context cropped to `max_seq_len`; `parameters()` order is token_emb,
positional (if learned), blocks, final_ln, head; `no_decay_params()` is every LayerNorm
parameter plus the ffn1 / ffn2 / out_proj biases.

Extension: `pos="learned"` selects a LearnedPE table (the reference always uses the fixed
sinusoidal table).  On CUDA the token gather and the positional add are one kernel, and the
head weight is stored with its row padded to a multiple of 8 columns so TMA can address the
50257-wide vocabulary (checkpoints still hold the unpadded [embed, vocab] matrix).  Without
gradients and in bf16 a forward is one native call, and `generate` is a prefill plus one
persistent kernel over cached keys and values (csrc/kernels/gpt_infer.cu); once the context
has to be cropped, every position changes and each token takes a full forward.
"""
from __future__ import annotations

import math
from typing import List, Optional

import torch

from .. import _backend as B
from ..utils import debug as _debug
from .. import autograd
from ..nn.dropout import Dropout
from ..nn.embedding import Embedding, embedding_backward_into
from ..nn.layernorm import LayerNorm
from ..nn.linear import Linear
from ..nn.module import Module
from ..nn.multihead import FlashMultiHeadAttention
from ..nn.positional import LearnedPE, SinusoidalPE, positional_backward_into
from ..nn.transformer import TransformerBlock
from ..tensor import Tensor


class GPT(Module):
    def __init__(self, vocab_size: int, embed_dim: int, num_heads: int, num_layers: int,
                 max_seq_len: int, dropout: Optional[float] = 0.1, pos: str = "sinusoidal"):
        dropout = 0.1 if dropout is None else dropout
        self.vocab_size = vocab_size
        self.embed_dim = embed_dim
        self.num_heads = num_heads
        self.num_layers = num_layers
        self.max_seq_len = max_seq_len
        self.token_emb = Embedding(vocab_size, embed_dim)
        self.pos_enc = (LearnedPE(max_seq_len, embed_dim) if pos == "learned"
                        else SinusoidalPE(max_seq_len, embed_dim))
        self.emb_drop = Dropout(dropout)
        self.blocks: List[TransformerBlock] = [
            TransformerBlock(embed_dim, num_heads, dropout) for _ in range(num_layers)]
        self.final_ln = LayerNorm(embed_dim)
        self.head = Linear(embed_dim, vocab_size, False, pad_out=True)
        self.training = True

    # ------------------------------------------------------------------ forward
    def _embed(self, ids: torch.Tensor, seq_len: int) -> Tensor:
        w = self.token_emb.weight
        if w._t.is_cuda:
            if not ids.is_cuda:
                ids = ids.cuda()
            ids = B._labels(ids)
            table = w._compute if w._compute is not None else w._t
            learned = isinstance(self.pos_enc, LearnedPE)
            if learned:
                pw = self.pos_enc.weight
                pos_table = pw._compute if (pw._compute is not None and
                                            pw._compute.dtype == table.dtype) else pw._t.to(table.dtype)
            else:
                pos_table = self.pos_enc._table(table)
            y, err = B.ext().embedding_forward(table, ids, pos_table, seq_len)
            _debug.check_index_word(err, "GPT token embedding: token id")
            out = Tensor(_data=y)
            batch = ids.numel() // seq_len
            pos_enc = self.pos_enc

            def grad_fn(g):
                if w.requires_grad:
                    embedding_backward_into(w, g._t, ids)
                if learned and pos_enc.weight.requires_grad:
                    positional_backward_into(pos_enc.weight, g._t, batch, seq_len)

            autograd.record("embed_tokens", [w, pos_enc.weight if learned else None], out, grad_fn)
            return out
        x = self.token_emb(Tensor(_data=ids))
        return self.pos_enc(x, seq_len)

    # ------------------------------------------------------------------ inference
    def _is_stock(self) -> bool:
        """Whether nobody has put code of their own between the layers: every layer is of the type
        the constructor makes, and no `forward`, `__call__` or `_embed` has been replaced, neither
        on a class nor on an instance."""
        if any(c.forward is not f or c.__call__ is not _CALL for c, f in _STOCK.items()):
            return False
        if type(self)._embed is not _EMBED or "_embed" in self.__dict__:
            return False
        pos = LearnedPE if type(self.pos_enc) is LearnedPE else SinusoidalPE
        layers = [(self.token_emb, Embedding), (self.pos_enc, pos), (self.emb_drop, Dropout),
                  (self.final_ln, LayerNorm), (self.head, Linear)]
        for b in self.blocks:
            if type(b) is not TransformerBlock:
                return False
            layers += [(b, TransformerBlock), (b.ln1, LayerNorm), (b.attn, FlashMultiHeadAttention),
                       (b.drop1, Dropout), (b.ln2, LayerNorm), (b.ffn1, Linear), (b.ffn2, Linear), (b.drop2, Dropout)]
            if type(b.attn) is FlashMultiHeadAttention:
                layers.append((b.attn.out_proj, Linear))
        for m, c in layers:
            if type(m) is not c or "forward" in m.__dict__:
                return False
        return True

    def _inference_weights(self):
        """The bf16 tensors the native inference path reads, or None where it does not apply
        (CPU, fp32 compute, active dropout, other head sizes, layers that are not the stock ones)."""
        if not self._is_stock():      # first: layers of other types have other attributes
            return None
        emb = self.token_emb.weight
        if not emb._t.is_cuda:
            return None

        def view(p):
            t = p._compute if p._compute is not None else p._t
            return t if t.dtype == torch.bfloat16 and t.is_contiguous() else None

        if view(emb) is None or self.embed_dim // self.num_heads not in (64, 128):
            return None
        if isinstance(self.pos_enc, LearnedPE):
            pos = view(self.pos_enc.weight)
        else:
            pos = self.pos_enc._table(view(emb))
        head = self.head.weight_storage if self.head.weight_storage is not None else self.head.weight
        ln = self.final_ln
        out = [view(emb), pos, view(ln.gamma), view(ln.beta), view(head)]
        if self.emb_drop.training and self.emb_drop.p > 0.0 or self.head.use_bias:
            return None
        scale = 1.0 / math.sqrt(self.embed_dim // self.num_heads)
        for b in self.blocks:
            a = b.attn
            if (not a.causal or a.num_heads != self.num_heads or a.scale != scale
                    or b.ln1.eps != ln.eps or b.ln2.eps != ln.eps
                    or b.training and (b.drop1.p > 0.0 or b.drop2.p > 0.0)
                    or not (a.out_proj.use_bias and b.ffn1.use_bias and b.ffn2.use_bias)):
                return None
            out += [view(b.ln1.gamma), view(b.ln1.beta), view(a.qkv_weight), view(a.out_proj.weight),
                    view(a.out_proj.bias), view(b.ln2.gamma), view(b.ln2.beta), view(b.ffn1.weight),
                    view(b.ffn1.bias), view(b.ffn2.weight), view(b.ffn2.bias)]
        if not 0 < len(self.blocks) <= 96 or any(t is None for t in out) or out[4].shape[1] % 8:
            return None
        # every block alike: the kernels take one set of widths, and vocab_size for table and head
        E, F = self.embed_dim, self.blocks[0].ffn1.out_features
        if (out[0].shape != (self.vocab_size, E) or out[1].shape[1:] != (E,) or out[2].shape != (E,)
                or out[3].shape != (E,) or self.head.out_features != self.vocab_size or out[4].shape[0] != E):
            return None
        widths = [(E,), (E,), (E, 3 * E), (E, E), (E,), (E,), (E,), (E, F), (F,), (F, E), (E,)]
        if F % 8 or [t.shape for t in out[5:]] != widths * len(self.blocks):
            return None
        return out

    def _decode_applies(self, w, temperature) -> bool:
        """Whether the decode kernel stands for a loop over `forward`: nobody has replaced that
        method, the model fits the kernel's shared memory, its weights allow 16-byte loads, the
        temperature keeps the order of the logits, and nobody asked for the checks that follow every launch."""
        return (getattr(self.forward, "__func__", None) is _FORWARD and not _debug._on
                and 0.0 < temperature < math.inf
                and all(t.data_ptr() % 16 == 0 for t in w)
                and B.ext().gpt_decode_fits(self.embed_dim, w[5 + 7].shape[1],
                                            self.embed_dim // self.num_heads, self.vocab_size))

    def forward(self, input: Tensor) -> Tensor:
        shape = input.shape
        seq_len = shape[1] if len(shape) >= 2 else shape[0]
        if not autograd.enabled and seq_len <= self.max_seq_len:
            w = self._inference_weights()
            if w is not None:
                ids = input._t.reshape(-1)
                ids = B._labels(ids if ids.is_cuda else ids.cuda())
                logits, err = B.ext().gpt_forward(w, self.num_heads, self.vocab_size, self.final_ln.eps,
                                                  ids, ids.numel() // seq_len, seq_len)
                _debug.check_index_word(err, "GPT token embedding: token id")
                if _debug._on:
                    _debug.check_kernels(B.ext())
                return Tensor(_data=logits[:, :self.vocab_size])
        x = self._embed(input._t.reshape(-1), seq_len)
        x = self.emb_drop(x)
        for block in self.blocks:
            x = block(x, seq_len)
        x = self.final_ln(x)
        return self.head(x)

    # ------------------------------------------------------------------ sampling
    def generate(self, prompt: Tensor, max_tokens: int = 100, temperature: float = 1.0,
                 top_k: int = 0) -> Tensor:
        temperature = 1.0 if temperature is None else temperature
        top_k = top_k or 0
        was_training = self.training
        self.eval()
        # a Tensor of token ids (as in the reference) or any plain sequence of ints
        src = prompt._t if isinstance(prompt, Tensor) else torch.as_tensor(prompt)
        tokens = [int(v) for v in src.reshape(-1).tolist()]
        dev = self.token_emb.weight._t.device
        gen = B.cpu_generator()
        todo = max_tokens or 100
        with autograd.no_grad():
            w = self._inference_weights()
            # cached keys and values serve until the context has to be cropped
            n = min(todo, self.max_seq_len - len(tokens) + 1)
            if w is not None and n > 0 and tokens and self._decode_applies(w, temperature):
                rnd = torch.rand(n, generator=gen).to(dev)
                ids = torch.tensor(tokens, dtype=torch.int32).to(dev)
                got = B.ext().gpt_generate(w, self.num_heads, self.vocab_size, self.final_ln.eps, ids, rnd,
                                           float(temperature), int(top_k)).tolist()
                if got.pop() != 0:
                    raise RuntimeError("GPT.generate: a grid-wide wait of the decode kernel ran out of time")
                tokens += got
                todo -= n
            for _ in range(todo):
                ctx = tokens[-self.max_seq_len:]
                inp = Tensor(_data=torch.tensor(ctx, dtype=torch.float32, device=dev).reshape(1, -1))
                autograd.zero_graph()
                logits = self.forward(inp)
                last = logits._t[len(ctx) - 1, :self.vocab_size].float().cpu()
                if temperature != 1.0:
                    last = last / temperature
                if 0 < top_k < self.vocab_size:
                    thresh = torch.topk(last, top_k).values[-1]
                    last = torch.where(last < thresh, torch.full_like(last, -math.inf), last)
                probs = torch.softmax(last, 0)
                r = torch.rand((), generator=gen).item()
                idx = int(torch.searchsorted(torch.cumsum(probs, 0), torch.tensor(r)).clamp(max=self.vocab_size - 1))
                tokens.append(idx)
        if was_training:
            self.train()
        return Tensor(_data=torch.tensor(tokens, dtype=torch.float32))

    # ------------------------------------------------------------------ protocol
    def children(self):
        return [self.token_emb, self.pos_enc, self.emb_drop, *self.blocks, self.final_ln, self.head]

    def parameters(self):
        params = list(self.token_emb.parameters())
        params.extend(self.pos_enc.parameters())
        for b in self.blocks:
            params.extend(b.parameters())
        params.extend(self.final_ln.parameters())
        params.extend(self.head.parameters())
        return params

    def no_decay_params(self):
        nd = list(self.final_ln.parameters())
        for b in self.blocks:
            nd.extend(b.ln1.parameters())
            nd.extend(b.ln2.parameters())
            for lin in (b.ffn1, b.ffn2, b.attn.out_proj):
                if lin.use_bias:
                    nd.append(lin.bias)
        return nd

    def __repr__(self):
        return "GPT(vocab=%d, embed=%d, heads=%d, layers=%d, max_seq=%d, params=%d)" % (
            self.vocab_size, self.embed_dim, self.num_heads, self.num_layers, self.max_seq_len,
            self.num_params())


# What the native inference path stands for: the methods as they are defined, see GPT._is_stock.
_CALL = Module.__call__
_EMBED, _FORWARD = GPT._embed, GPT.forward
_STOCK = {c: c.forward for c in (Embedding, LearnedPE, SinusoidalPE, Dropout, LayerNorm, Linear,
                                 FlashMultiHeadAttention, TransformerBlock)}
