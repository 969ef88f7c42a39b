// A whole chunk of a prompt in one host call: embedding rows, then per layer five launches, then the final norm. The launches are
// issued from here and not from Python because a short prompt is bound by them: 242 calls through ctypes took 2.7 ms for 77 tokens,
// more than the GPU needs.
#include "prefill.h"
#include "common.cuh"
#include "umma.cuh"

namespace b200 {

namespace {

// x[t] = emb[ids[t]]; an id outside the table reads row 0 (embed_row_kernel). xw and sums as the GEMMs leave them (PrefillNorm), but with a
// power of two for every row, which takes its largest |x * w| to 2^13 .. 2^14: the row is final here, and embeddings may be small.
__global__ void __launch_bounds__(256)
embed_rows_kernel(const uint4* __restrict__ emb, const long long* __restrict__ ids, const uint4* __restrict__ w, uint4* __restrict__ x,
                  uint4* __restrict__ xw, float* __restrict__ ss_out, float* __restrict__ inv_out, int nchunk, int parts, int V) {
  __shared__ float part[8], top[8];
  pdl_wait();
  // behind the wait: no kernel of the chunk starts before what precedes the chunk has completed, so each of them may read what the
  // chunk's kernels do not write (weights, positions, block table) ahead of its own wait
  pdl_launch_dependents();
  long long t = ids[blockIdx.x];
  if (t < 0 || t >= V) t = 0;
  emb += (size_t)t * nchunk, x += (size_t)blockIdx.x * nchunk, xw += (size_t)blockIdx.x * nchunk;
  float ss = 0.f, mx = 0.f;
  for (int i = threadIdx.x; i < nchunk; i += blockDim.x) {
    const uint4 r = __ldg(emb + i);
    x[i] = r;
    float f[8], g[8];
    unpack8(r, f);
    unpack8(__ldg(w + i), g);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss = fmaf(f[k], f[k], ss), mx = fmaxf(mx, fabsf(f[k] * g[k]));
  }
  ss = warp_sum(ss), mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss, top[threadIdx.x >> 5] = mx;
  __syncthreads();
  ss = 0.f;
  for (int k = 0; k < 8; ++k) ss += part[k], mx = fmaxf(mx, top[k]);
  const float inv = umma::pow2_above(mx) * 0x1p-14f, scale = 1.f / inv;
  for (int i = threadIdx.x; i < nchunk; i += blockDim.x) {
    float f[8], g[8];
    unpack8(__ldg(emb + i), f);
    unpack8(__ldg(w + i), g);
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = as_u32(__floats2half2_rn(f[2 * k] * g[2 * k] * scale, f[2 * k + 1] * g[2 * k + 1] * scale));
    xw[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  for (int i = threadIdx.x; i < parts; i += blockDim.x) ss_out[(size_t)blockIdx.x * parts + i] = i == 0 ? ss : 0.f;
  if (threadIdx.x == 0) inv_out[blockIdx.x] = inv;
}

}  // namespace

cudaError_t prefill_chunk_dispatch(const PrefillParams& p, cudaStream_t st) {
#define TRY(call)                        \
  do {                                   \
    const cudaError_t e_ = (call);       \
    if (e_ != cudaSuccess) return e_;    \
  } while (0)
  const int n_qkv = (p.n_q + 2 * p.n_kv) * p.D, n_att = p.n_q * p.D, parts = p.H / 128;
  // the residual rows' sums and factors, in front of attention (a) and of the MLP (m): in the buffer that only the last down projection
  // still writes as rows (16 bytes and more per 128 columns are there for 8 and 8 a token)
  float *ss_a = (float*)p.o, *ss_m = ss_a + (size_t)p.T * parts, *inv_a = ss_m + (size_t)p.T * parts, *inv_m = inv_a + p.T;
  const float inv_h = 1.f / (float)p.H;
  half *x = (half*)p.x, *xw = (half*)p.normed;
  B200_LAUNCH(embed_rows_kernel, dim3(p.T), dim3(256), 0, st, (const uint4*)p.emb, p.ids, (const uint4*)p.layers[0].ln1, (uint4*)p.x,
              (uint4*)p.normed, ss_a, inv_a, p.H >> 3, parts, p.V);
  for (int l = 0; l < p.L; ++l) {
    const StepLayer& ly = p.layers[l];
    const bool last = l + 1 == p.L;
    const PrefillNorm at_qkv = {ss_a, inv_a, nullptr, nullptr, nullptr, nullptr, nullptr, parts, inv_h, p.eps};
    const PrefillNorm to_mlp = {nullptr, nullptr, x, xw, ly.ln2, ss_m, inv_m, parts, inv_h, p.eps};
    const PrefillNorm at_mlp = {ss_m, inv_m, nullptr, nullptr, nullptr, nullptr, nullptr, parts, inv_h, p.eps};
    const PrefillNorm to_next = {nullptr, nullptr, x, xw, last ? nullptr : p.layers[l + 1].ln1, ss_a, inv_a, parts, inv_h, p.eps};
    const PrefillRope rope = {p.cos_t, p.sin_t, p.pos, p.bt, ly.kc, ly.vc, p.n_q, p.n_kv, p.D, p.log2P};
    TRY(prefill_gemm_tiled_dispatch(ly.w[0], p.normed, p.qkv, p.T, n_qkv, p.H, 0, 0, &at_qkv, &rope, st));
    TRY(prefill_attention_dispatch(p.qkv, n_qkv, ly.kc, ly.vc, p.bt, p.start, p.T, p.n_q, p.n_kv, p.D, p.log2P, p.attn, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[1], p.attn, nullptr, p.T, p.H, n_att, 0, 0, &to_mlp, nullptr, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[2], p.normed, p.act, p.T, p.I, p.H, 1, 0, &at_mlp, nullptr, st));
    TRY(prefill_gemm_tiled_dispatch(ly.w[3], p.act, p.o, p.T, p.H, p.I, 0, 0, last ? nullptr : &to_next, nullptr, st));
  }
  return add_rmsnorm_dispatch(p.x, p.o, p.norm_f, p.normed, p.T, p.H, p.eps, st);
#undef TRY
}

}  // namespace b200
