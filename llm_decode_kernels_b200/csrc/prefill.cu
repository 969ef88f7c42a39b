// A whole chunk of a prompt in one host call: embedding rows, then per layer eight launches, then the final norm. The launches are
// issued from here and not from Python because a short prompt is bound by them: 242 calls through ctypes took 2.7 ms for 77 tokens,
// more than the GPU needs.
#include "prefill.h"
#include "common.cuh"

namespace b200 {

namespace {

// x[t] = emb[ids[t]]; an id outside the table reads row 0 (embed_row_kernel)
__global__ void embed_rows_kernel(const uint4* __restrict__ emb, const long long* __restrict__ ids, uint4* __restrict__ x, int nchunk,
                                  int V) {
  pdl_launch_dependents();
  pdl_wait();
  long long t = ids[blockIdx.x];
  if (t < 0 || t >= V) t = 0;
  for (int i = threadIdx.x; i < nchunk; i += blockDim.x) x[(size_t)blockIdx.x * nchunk + i] = emb[(size_t)t * nchunk + i];
}

}  // namespace

cudaError_t prefill_chunk_dispatch(const PrefillParams& p, cudaStream_t st) {
#define TRY(call)                        \
  do {                                   \
    const cudaError_t e_ = (call);       \
    if (e_ != cudaSuccess) return e_;    \
  } while (0)
  const int n_qkv = (p.n_q + 2 * p.n_kv) * p.D, n_att = p.n_q * p.D;
  B200_LAUNCH(embed_rows_kernel, dim3(p.T), dim3(256), 0, st, (const uint4*)p.emb, p.ids, (uint4*)p.x, p.H >> 3, p.V);
  const void* delta = nullptr;
  for (int l = 0; l < p.L; ++l) {
    const StepLayer& ly = p.layers[l];
    TRY(add_rmsnorm_dispatch(p.x, delta, ly.ln1, p.normed, p.T, p.H, p.eps, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[0], p.normed, p.qkv, p.T, n_qkv, p.H, 0, 0, st));
    TRY(rope_append_dispatch(p.qkv, p.cos_t, p.sin_t, p.pos, p.bt, 0, ly.kc, ly.vc, p.T, p.n_q, p.n_kv, p.D, p.log2P, st));
    TRY(prefill_attention_dispatch(p.qkv, n_qkv, ly.kc, ly.vc, p.bt, p.start, p.T, p.n_q, p.n_kv, p.D, p.log2P, p.attn, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[1], p.attn, p.o, p.T, p.H, n_att, 0, 0, st));
    TRY(add_rmsnorm_dispatch(p.x, p.o, ly.ln2, p.normed, p.T, p.H, p.eps, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[2], p.normed, p.act, p.T, p.I, p.H, 1, 0, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[3], p.act, p.o, p.T, p.H, p.I, 0, 0, st));
    delta = p.o;
  }
  return add_rmsnorm_dispatch(p.x, delta, p.norm_f, p.normed, p.T, p.H, p.eps, st);
#undef TRY
}

}  // namespace b200
