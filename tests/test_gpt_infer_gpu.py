"""Native GPT inference (csrc/kernels/gpt_infer.cu) against the layer-by-layer path.

The scoring forward issues the same kernels as the layers, so its logits are the same bits.  The
decode kernel takes its sums in another order and keeps attention weights in fp32: a token it
draws must lie within reach of the uniform number under the layer path's distribution for the
same prefix, i.e. cdf(token - 1) - d <= r <= cdf(token) + d.  The logits here are below 16 in size
and bf16, each off by at most an ulp or two (2 * 2^-5), so a cdf value p (1 - p) moves by at most
0.25 * 2 * 2^-4 < d = 0.04."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(vocab, embed, heads, layers, max_seq, pos):
    import luatorch_b200 as lf
    lf.manual_seed(11)
    m = lf.models.GPT(vocab, embed, heads, layers, max_seq, 0.0, pos=pos)
    g = torch.Generator().manual_seed(3)
    for b in m.blocks:
        for lin in (b.attn.out_proj, b.ffn1, b.ffn2):
            lin.bias._t.copy_(torch.randn(lin.bias._t.shape, generator=g) * 0.1)
        for ln in (b.ln1, b.ln2):
            ln.gamma._t.copy_(1 + 0.1 * torch.randn(ln.gamma._t.shape, generator=g))
            ln.beta._t.copy_(0.1 * torch.randn(ln.beta._t.shape, generator=g))
        for lin in (b.attn.out_proj, b.ffn2):
            lin.weight._t.mul_((2 * layers) ** -0.5)
    m.head.weight._t.mul_(0.5)
    lf.cuda.amp.autocast_bf16(m)
    return m.eval()


def _layerwise(m, ids):
    import luatorch_b200 as lf
    native, m._inference_weights = m._inference_weights, lambda: None
    try:
        with lf.autograd.no_grad():
            return m.forward(lf.Tensor.wrap(ids))._t
    finally:
        m._inference_weights = native


@pytest.mark.parametrize("batch,seq", [(1, 1), (3, 77), (2, 128)])
@pytest.mark.parametrize("embed,heads", [(128, 2), (256, 2)])
def test_scoring_forward_is_the_layers(batch, seq, embed, heads):
    import luatorch_b200 as lf
    m = _model(331, embed, heads, 2, 128, "learned")
    ids = torch.randint(0, 331, (batch, seq), device="cuda", dtype=torch.int32)
    assert m._inference_weights() is not None
    with lf.autograd.no_grad():
        got = m.forward(lf.Tensor.wrap(ids))._t
    assert got.shape == (batch * seq, 331)
    assert torch.equal(got, _layerwise(m, ids))


@pytest.mark.parametrize("vocab,embed,heads,layers,pos,prompt,n,temperature,top_k", [
    (50257, 768, 12, 2, "learned", 100, 12, 0.8, 40),
    (1000, 256, 4, 2, "sinusoidal", 17, 12, 1.0, 0),       # whole vocabulary
    (777, 192, 3, 3, "learned", 1, 16, 1.3, 300),          # more than one CTA maximum per rank
    (50257, 128, 2, 1, "learned", 250, 12, 1.0, 5000),     # across the fused-attention limit (256 keys)
    (97, 64, 1, 1, "learned", 3, 9, 0.7, 5),               # fewer units than CTAs
    (500, 256, 2, 2, "learned", 120, 14, 1.0, 20),         # head dim 128, across its limit (128 keys)
    (333, 1280, 20, 1, "learned", 40, 6, 1.0, 50),         # more heads than K slices, wide residual
])
def test_decode_draws_from_the_layers_distribution(vocab, embed, heads, layers, pos, prompt, n, temperature, top_k):
    import luatorch_b200 as lf
    m = _model(vocab, embed, heads, layers, 300, pos)
    ids = [(37 * i + 11) % vocab for i in range(prompt)]
    lf.manual_seed(5)
    toks = [int(t) for t in m.generate(ids, n, temperature, top_k).tolist()]
    lf.manual_seed(5)
    assert [int(t) for t in m.generate(ids, n, temperature, top_k).tolist()] == toks
    assert toks[:prompt] == ids and len(toks) == prompt + n
    lf.manual_seed(5)
    rnd = torch.rand(n, generator=lf._backend.cpu_generator()).tolist()
    full = torch.tensor([toks], dtype=torch.int32, device="cuda")
    logits = _layerwise(m, full)[prompt - 1:-1].double() / temperature
    for i in range(n):
        v = logits[i]
        if 0 < top_k < vocab:
            v = torch.where(v < torch.topk(v, top_k).values[-1], torch.full_like(v, -float("inf")), v)
        cdf = torch.cumsum(torch.softmax(v, 0), 0)
        t = toks[prompt + i]
        lo = float(cdf[t - 1]) if t else 0.0
        assert lo - 0.04 <= rnd[i] <= float(cdf[t]) + 0.04, (i, t, lo, rnd[i], float(cdf[t]))
        if 0 < top_k < vocab:       # and it is among the top_k: two logits, two ulps of 2^-4 each
            assert float(logits[i][t]) >= float(torch.topk(logits[i], top_k).values[-1]) - 0.25 / temperature


def test_decode_kernel_only_stands_for_the_stock_loop():
    """Models and options that the decode kernel does not cover keep the loop over `forward`."""
    import luatorch_b200 as lf
    from luatorch_b200 import _C
    calls = []

    class Counting(lf.models.GPT):
        def forward(self, x):
            calls.append(x.shape)
            return super().forward(x)

    class Scaled(lf.nn.Linear):
        def forward(self, *args, **kwargs):
            calls.append(None)
            return super().forward(*args, **kwargs)

    def seen(m, temperature=1.0):
        calls.clear()
        out = m.generate([1, 2, 3], 3, temperature, 5)
        assert out.shape == [6] and all(0 <= int(t) < 97 for t in out.tolist())
        return len(calls)

    m = Counting(97, 128, 2, 1, 24, 0.0)
    lf.cuda.amp.autocast_bf16(m)
    assert seen(m.eval()) == 3
    m = _model(97, 128, 2, 1, 24, "learned")
    assert seen(m) == 0 and m._inference_weights() is not None
    w = m._inference_weights()
    assert not m._decode_applies(w, -1.0) and not m._decode_applies(w, 0.0) and not m._decode_applies(w, float("nan"))
    assert m._decode_applies(w, 0.5)
    assert seen(m, -1.0) == 0                                 # the loop, over the stock forward
    m.blocks[0].ffn1.__class__ = Scaled
    assert m._inference_weights() is None and seen(m) == 3
    # 24 bytes of shared memory per embedding column beside 100 KB of weight slots
    assert _C.gpt_decode_fits(4096, 16384, 128, 50257) and not _C.gpt_decode_fits(4608, 18432, 128, 50257)


def test_context_longer_than_the_model():
    """Past max_seq_len the context is cropped and every token takes a forward of its own."""
    import luatorch_b200 as lf
    m = _model(97, 64, 1, 1, 24, "learned")
    out = m.generate(list(range(20)), 12, 1.0, 3)
    assert out.shape == [32] and all(0 <= int(t) < 97 for t in out.tolist())


def _same_as_layers(m, ids):
    """The forward without gradients gives what the loop over the layers gives."""
    import luatorch_b200 as lf
    with lf.autograd.no_grad():
        got = m.forward(lf.Tensor.wrap(ids))._t
    return torch.equal(got, _layerwise(m, ids))


LAYERS = {"block": lambda m: m.blocks[1], "attn": lambda m: m.blocks[0].attn, "out_proj": lambda m: m.blocks[1].attn.out_proj,
          "ln2": lambda m: m.blocks[0].ln2, "ffn1": lambda m: m.blocks[1].ffn1, "ffn2": lambda m: m.blocks[0].ffn2,
          "emb_drop": lambda m: m.emb_drop, "final_ln": lambda m: m.final_ln,
          "head": lambda m: m.head}


@pytest.mark.parametrize("where", ["instance", "class"])
@pytest.mark.parametrize("layer", list(LAYERS))
def test_a_replaced_forward_is_called(layer, where, monkeypatch):
    """Scoring and sampling call what a program has put in a layer's place."""
    import luatorch_b200 as lf
    m = _model(97, 128, 2, 2, 24, "learned")
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    target = LAYERS[layer](m)
    stock, seen = target.forward, []

    def doubled(*args, **kwargs):
        seen.append(1)
        if where == "class":
            out = original(*args, **kwargs)
        else:
            out = stock(*args, **kwargs)
        return lf.Tensor(_data=out._t * 2)

    if where == "class":
        owner = next(c for c in type(target).__mro__ if "forward" in vars(c))
        original = owner.forward
        monkeypatch.setattr(owner, "forward", doubled)
    else:
        target.forward = doubled
    assert _same_as_layers(m, ids) and seen
    seen.clear()
    assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6] and len(seen) >= 3


def test_a_replaced_call_or_embedding_is_called(monkeypatch):
    import luatorch_b200 as lf
    seen = []

    class Shifted(lf.models.GPT):
        def _embed(self, ids, seq_len):
            seen.append(seq_len)
            return super()._embed((ids.int() + 1) % 97, seq_len)

    lf.manual_seed(2)
    m = Shifted(97, 128, 2, 1, 24, 0.0)
    lf.cuda.amp.autocast_bf16(m)
    m.eval()
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    assert _same_as_layers(m, ids) and len(seen) == 2
    m = _model(97, 128, 2, 1, 24, "learned")
    call = lf.nn.Module.__call__
    monkeypatch.setattr(lf.nn.Module, "__call__", lambda self, *a, **k: (seen.append(type(self)), call(self, *a, **k))[1])
    seen.clear()
    assert _same_as_layers(m, ids) and lf.nn.Linear in seen
    seen.clear()
    m.generate([1, 2, 3], 2, 1.0, 5)
    assert lf.nn.LayerNorm in seen


@pytest.mark.parametrize("what", ["head", "final_ln", "pos_enc", "emb_drop", "block", "attn"])
def test_layers_of_other_types(what):
    """A module of the program's own in a layer's place: the loop over the layers, whatever it has inside."""
    import luatorch_b200 as lf
    nn = lf.nn

    class Own(nn.Module):                       # has none of the stock layers' attributes
        def __init__(self, fn):
            self.fn = fn

        def forward(self, x, *args, **kwargs):
            return self.fn(x, *args, **kwargs)

    m = _model(97, 128, 2, 2, 24, "sinusoidal")
    if what == "block":
        m.blocks[1] = Own(lambda x, s: x)
    elif what == "attn":
        m.blocks[0].attn = Own(lambda x, seq_len=None, residual=None: residual)
    elif what == "pos_enc":
        stock = _model(97, 128, 2, 2, 24, "sinusoidal")
        m.pos_enc, m._embed = Own(None), stock._embed
    else:
        stock = getattr(m, what)
        setattr(m, what, Own(lambda x: stock(x)))
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    assert _same_as_layers(m, ids)
    assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6]


@pytest.mark.parametrize("widths", [(4, 2), (2, 4), (1, 3)])
def test_blocks_of_different_width(widths):
    import luatorch_b200 as lf
    lf.manual_seed(4)
    m = lf.models.GPT(97, 128, 2, 2, 24, 0.0, pos="learned")
    m.blocks = [lf.nn.TransformerBlock(128, 2, 0.0, w) for w in widths]
    lf.cuda.amp.autocast_bf16(m)
    m.eval()
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    assert _same_as_layers(m, ids)
    assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6]


def test_feed_forward_width_that_is_no_multiple_of_eight():
    import luatorch_b200 as lf
    lf.manual_seed(4)
    m = lf.models.GPT(97, 128, 2, 1, 24, 0.0, pos="learned")
    m.blocks[0].ffn1, m.blocks[0].ffn2 = lf.nn.Linear(128, 100), lf.nn.Linear(100, 128)
    lf.cuda.amp.autocast_bf16(m)
    m.eval()
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    assert _same_as_layers(m, ids)
    assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6]


def test_a_model_without_blocks():
    import luatorch_b200 as lf
    m = _model(97, 128, 2, 0, 24, "learned")
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    assert _same_as_layers(m, ids)
    assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6]


def test_table_and_head_of_other_widths():
    """An embedding with more rows than `vocab_size`, a head with fewer or more columns."""
    import luatorch_b200 as lf
    for rows, cols in ((120, 97), (97, 40), (97, 128)):
        lf.manual_seed(4)
        m = lf.models.GPT(97, 128, 2, 1, 24, 0.0, pos="learned")
        m.token_emb, m.head = lf.nn.Embedding(rows, 128), lf.nn.Linear(128, cols, False, pad_out=True)
        lf.cuda.amp.autocast_bf16(m)
        m.eval()
        ids = torch.tensor([[0, 5, rows - 1, 7]], device="cuda", dtype=torch.int32)
        with lf.autograd.no_grad():
            assert m.forward(lf.Tensor.wrap(ids)).shape == [4, cols]
        assert _same_as_layers(m, ids)
        assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6]


@pytest.mark.parametrize("name", ["ffn1", "ffn2", "out_proj", "qkv"])
def test_weights_off_the_16_byte_grid(name):
    """bf16 weights that are a view at an odd offset: the decode kernel's 16-byte loads cannot take them."""
    import luatorch_b200 as lf
    from luatorch_b200 import _C
    m = _model(97, 128, 2, 2, 24, "learned")
    b = m.blocks[1]
    p = {"ffn1": b.ffn1.weight, "ffn2": b.ffn2.weight, "out_proj": b.attn.out_proj.weight, "qkv": b.attn.qkv_weight}[name]
    t = p._compute
    buf = torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)
    p._compute = buf[1:].view(t.shape).copy_(t)
    w = m._inference_weights()
    assert w is not None and not m._decode_applies(w, 1.0)
    with pytest.raises(RuntimeError, match="16 bytes"):
        _C.gpt_generate(w, 2, 97, 1e-5, torch.zeros(3, device="cuda", dtype=torch.int32), torch.rand(2, device="cuda"), 1.0, 5)
    ids = torch.arange(5, device="cuda", dtype=torch.int32).reshape(1, 5)
    assert _same_as_layers(m, ids)
    assert m.generate([1, 2, 3], 3, 1.0, 5).shape == [6]


def _exact_model(vocab, embed):
    """One block that adds nothing, embeddings of +-1 that LayerNorm leaves as they are, a head of
    multiples of 1/16: every logit is exact in fp32 whatever the order of the sums."""
    import luatorch_b200 as lf
    lf.manual_seed(1)
    m = lf.models.GPT(vocab, embed, embed // 64, 1, 64, 0.0, pos="learned")
    g = torch.Generator().manual_seed(vocab)
    m.pos_enc.weight._t.zero_()
    for lin in (m.blocks[0].attn.out_proj, m.blocks[0].ffn2):
        lin.weight._t.zero_()
    signs = torch.ones(embed)
    signs[:embed // 2] = -1
    order = torch.rand(vocab, embed, generator=g).argsort(1)
    m.token_emb.weight._t.copy_(signs[order])
    m.head.weight._t.copy_(torch.randint(-6, 7, (embed, vocab), generator=g) / 16.0)
    lf.cuda.amp.autocast_bf16(m)
    return m.eval()


@pytest.mark.parametrize("embed", [64, 128])           # 64: no room for a list of candidates
@pytest.mark.parametrize("vocab,top_k", [
    (777, 5), (777, 140),          # few candidates
    (2500, 148),                   # ties at the cut
    (777, 300), (9000, 5000),      # the threshold by bisection, runs of columns per thread
    (777, 0), (9000, 0), (50257, 0),
])
def test_decode_draws_the_exact_token(vocab, top_k, embed):
    """Known logits: the token is the one at the uniform number under their distribution, and a
    column that the cut has removed is never drawn, at the ends of the range of rnd either."""
    from luatorch_b200 import _C
    m = _exact_model(vocab, embed)
    w = m._inference_weights()
    assert m._decode_applies(w, 1.0)
    g = torch.Generator().manual_seed(7)
    rnd = torch.rand(30, generator=g)
    rnd[::5] = 0.0
    rnd[1::5] = 1 - 2.0 ** -24
    toks = [3] + _C.gpt_generate(w, embed // 64, vocab, m.final_ln.eps, torch.tensor([3], device="cuda", dtype=torch.int32),
                                 rnd.cuda(), 1.0, top_k).tolist()[:-1]
    logits = _layerwise(m, torch.tensor([toks], dtype=torch.int32, device="cuda"))[:-1].double().cpu()
    for i in range(30):
        v = logits[i]
        if top_k:
            v = torch.where(v < torch.topk(v, top_k).values[-1], torch.full_like(v, -float("inf")), v)
        p = torch.softmax(v, 0)
        cdf, t, r = torch.cumsum(p, 0), toks[i + 1], float(rnd[i])
        assert float(p[t]) > 0.0, (i, t)
        # fp32 sums of at most 50257 weights, expf to a few ulps: far below 1e-4 of the total
        lo = float(cdf[t] - p[t])
        assert lo - 1e-4 <= r <= float(cdf[t]) + 1e-4, (i, t, lo, r, float(cdf[t]))
        if abs(lo - r) > 1e-4 and abs(float(cdf[t]) - r) > 1e-4:
            assert t == int(torch.searchsorted(cdf, torch.tensor(r, dtype=torch.float64)))


@pytest.mark.parametrize("embed,ffn,batch,seq", [(2048, 8192, 1, 64), (2304, 2304, 1, 17), (2048, 8192, 3, 100), (128, 4104, 1, 200)])
def test_long_products_of_short_prompts_are_the_layers(embed, ffn, batch, seq):
    """Products that the layers cut along K are cut here too: the same bits."""
    import luatorch_b200 as lf
    lf.manual_seed(4)
    m = lf.models.GPT(97, embed, embed // 128, 1, 128, 0.0, pos="learned")
    m.blocks[0].ffn1, m.blocks[0].ffn2 = lf.nn.Linear(embed, ffn), lf.nn.Linear(ffn, embed)
    lf.cuda.amp.autocast_bf16(m)
    m.eval()
    assert m._inference_weights() is not None
    ids = torch.randint(0, 97, (batch, seq), device="cuda", dtype=torch.int32)
    assert _same_as_layers(m, ids)
