// Inference with a GPT decoder's bf16 weights: whole-sequence forward (scoring, prefill) and
// token-by-token sampling, without per-layer host work.  See gpt_infer.cu.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace lt {

constexpr int GPT_MAX_LAYERS = 96;

// bf16 device pointers; matrices are [in, out] with contiguous rows.
struct GptLayer {
  const void *ln1_g, *ln1_b, *wqkv, *wo, *bo, *ln2_g, *ln2_b, *w1, *b1, *w2, *b2;
};
struct GptWeights {
  int layers = 0, embed = 0, heads = 0, head_dim = 0, ffn = 0, vocab = 0;
  int64_t head_ld = 0;              // row stride of `head` (vocab padded to a multiple of 8)
  float eps = 1e-5f, scale = 0.125f;
  const void *tok = nullptr;        // [vocab, embed]
  const void *pos = nullptr;        // [>= positions, embed]
  const void *lnf_g = nullptr, *lnf_b = nullptr, *head = nullptr;
  GptLayer layer[GPT_MAX_LAYERS];
};

// Scratch of a forward over n tokens (bytes).
size_t gpt_forward_workspace(const GptWeights& w, int64_t n_tokens);
// Runs the blocks over ids [batch, seq] (id kinds as in ops.h) and leaves the residual stream
// [batch * seq, embed] in *x_out (inside `workspace`).  `cache`: optional [layers, cache_rows,
// 3 embed] that keeps every layer's q | k | v rows (batch 1).  `err`: status words of the gather.
cudaError_t gpt_forward(const GptWeights& w, const void* ids, int id_kind, int64_t batch, int64_t seq,
                        void* workspace, void* cache, int64_t cache_rows, int* err, void** x_out,
                        cudaStream_t s);
// logits [n, head_ld] = LayerNorm(x [n, embed]) head; `workspace` as gpt_forward's.
cudaError_t gpt_logits(const GptWeights& w, const void* x, int64_t n, void* workspace, void* logits,
                       cudaStream_t s);

// Sampling: token i of [first, last) is drawn from the logits after position prompt + i - 1 with
// temperature, top_k (<= 0: all) and the uniform number rnd[i]; ids_out[i] receives it.  `x`
// is the residual stream of the prompt's last position (used for i == 0), `cache` the prompt's
// q | k | v rows with room for the new ones.  `scratch`: gpt_decode_scratch() bytes.  status[0]
// is set when a grid-wide wait ran out of time.
// A model fits when its vectors do (shared memory) and table offsets stay below 2^31.
bool gpt_decode_fits(int64_t embed, int64_t ffn, int64_t head_dim, int64_t vocab);
size_t gpt_decode_scratch(const GptWeights& w);
cudaError_t gpt_decode(const GptWeights& w, const void* x, void* cache, int64_t cache_rows, int prompt,
                       int first, int last, float temperature, int top_k, const float* rnd, int* ids_out,
                       void* scratch, int* status, cudaStream_t s);

}  // namespace lt
