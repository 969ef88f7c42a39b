// Shared by the kernels of the prompt path.
#pragma once
#include "decode_step.h"
#include <cuda.h>
#include <cuda_runtime.h>

namespace b200 {

// Tensor map of activations X fp16 [T, K], 128-byte swizzle, zeros past T: coordinates (column in a 64-column chunk, token, chunk),
// boxes of 64 columns x box_rows tokens x chunks. False if the driver refuses (alignment).
bool encode_activation_map(CUtensorMap* map, const void* X, int T, int K, int box_rows, int chunks);

// RMSNorm inside the GEMMs of a prompt. The norm's factor is one number per token, so a GEMM may read rows that lack it and apply it to its
// outputs. What it reads is xw = fp16(x * w / p), written by the GEMM that finished the residual row x (RESIDUAL of
// prefill_gemm_tiled_kernel: x += its output) together with the sums of x^2 over each 128 columns.
// Range: p is the power of two that brings the largest |w| into [0.5, 1). |x * w / p| < 65504 then for every finite x, so nothing
// overflows however much a row grows in one addition, and small weights do not push a row among the subnormals. (A scale taken from
// the row as it was before the addition overflows where that addition makes it large.)
// Precision: one rounding, where w * fp16(x * factor) has two: a row is 2.07e-4 off instead of 2.9e-4. Products below 2^-14 are
// subnormal and keep 2^-25, as additions leave it in x; that is less than the two roundings keep where the products' root mean square
// is below 8e-5: rows of rms 1e-3 whose typical weight is below 0.08 p, rows of rms 1e-2 below 0.008 p. Embeddings, which may be
// so small, are scaled row by row (embed_rows_kernel).
struct PrefillNorm {
  const float* ss_in;    // [T][parts] sums of squares of the rows behind X, which are to be normalised
  const float* inv_in;   // [T] what X lacks beside the norm's factor (p)
  half *x, *xw;          // RESIDUAL: [T, N]; otherwise null
  const half* w;         // [N] the next norm's weight
  float *ss_out, *inv_out;
  int parts;             // H / 128
  float inv_h, eps;
};

// RoPE and the append to the paged cache inside the qkv GEMM (rope_append_rows_kernel's arithmetic on the fp16 outputs): q goes to Y
// rotated, k rotated and v as they are to the caches. A launch of its own for that was 1 us a layer at few tokens and 4 at 512. Whole prompt
// us, own launch / here: TinyLlama shape 8 tokens 829 / 782, 77 976 / 966, 512 1,631 / 1,598, 768 2,021 / 1,980, 1000 2,411 / 2,442, 1400 3,274 /
// 3,306, 2000 4,532 / 4,482, 4000 9,733 / 9,638; 8B shape (8 layers) 77 697 / 683, 1000 3,491 / 3,456, 4000 13,365 / 13,195; 70B shape (4 layers) 77
// 908 / 900, 1000 6,019 / 5,980, 4000 25,162 / 25,046. Behind only for TinyLlama at 900 to 1400 tokens (1 %: attention's CTAs, one wave there, started
// up beside the small launch), which is not worth a second form.
struct PrefillRope {
  const float *cos_t, *sin_t;   // [positions, D / 2]
  const int *pos, *bt;          // [T]; block table
  half *kc, *vc;                // null: no RoPE
  int n_q, n_kv, D, log2P;
};

// One chunk of a prompt: T tokens at positions start .. start + T - 1 of the sequence whose block table is bt.
struct PrefillParams {
  const StepLayer* layers;   // host array; matrices in tile layout, gate|up paired
  int L, H, I, n_q, n_kv, D, V, log2P;
  float eps;
  const void *emb, *norm_f;
  const float *cos_t, *sin_t;
  const int* bt;
  const long long* ids;      // [T]
  const int* pos;            // [T] start, start + 1, ...
  int T, start;
  void *x, *normed, *qkv, *attn, *o, *act;   // fp16 [T, H], [T, H], [T, (n_q + 2 n_kv) D], [T, n_q D], [T, H], [T, I]
};

cudaError_t prefill_chunk_dispatch(const PrefillParams& p, cudaStream_t st);
bool prefill_attention_takes(int D, int n_q, int n_kv);
cudaError_t prefill_attention_dispatch(const void* q, int q_stride, const void* kc, const void* vc, const int* bt, int start, int T,
                                       int n_q, int n_kv, int D, int log2P, void* out, cudaStream_t st);
cudaError_t prefill_attention_status(int* code);
// norm: null, or the norm of X's rows to apply, or (norm->x) the residual row to finish instead of storing Y. rope: null, or what the
// qkv GEMM does with its outputs.
cudaError_t prefill_gemm_tiled_dispatch(const void* Wt, const void* X, void* Y, int T, int N, int K, int swiglu, int force_split,
                                        const PrefillNorm* norm, const PrefillRope* rope, cudaStream_t st);
cudaError_t add_rmsnorm_dispatch(void* x, const void* delta, const void* w, void* out, int rows, int H, float eps,
                                 cudaStream_t st);

}  // namespace b200
