// Quantizer kernels of the INT4 format (quant.py states the format and holds the torch form these reproduce).
//
// quantize_w4_kernel: one pass from the weights to the kernel format. The torch form is ~15 elementwise and reduction
// kernels over fp32 and int64 copies of the matrix (with clipping: per factor), about 60 bytes of traffic per weight and
// pass; this reads the weight once and writes what was asked for. Bound by instruction issue: 133
// instructions a weight with clipping, 19 per candidate range (packed f32x2 arithmetic, a group's seven (scale, zero) worked out by seven
// of its lanes instead of by all sixteen), and the schedulers issue in 78 % of the cycles; without it 30, in 61 %.
//   11264 x 2048 fp16, group 128: with clipping 4,210 us in torch, 106 us here; without 28 us with the call around it.
// gptq_block_kernel: the sequential column loop of GPTQ inside one block of columns. The torch form launches ~14 kernels
// per COLUMN, each a few microseconds for a microsecond of work. Rows are independent of each other in GPTQ, so a warp takes a row:
// its part of the block lives in registers (four columns a lane), the block of the inverse Hessian's factor in shared
// memory, and a column costs one broadcast, the rounding, one division and four multiply-subtracts per lane. Bound by
// that dependent chain (~150 cycles a column), which the rows of a matrix hide behind each other.
//   2048 x 5632, 44 blocks with the update of the columns behind each: 560 ms as torch operators, 4.0 ms here.
//
// Both round exactly as the torch form does on a CUDA device: division by 15 as a product with the fp32 reciprocal,
// scale rounded to fp16 before use, correctly rounded quotients, round half to even, products and differences rounded
// separately, squared errors added four neighbours first and then pairwise. So levels, scales and zero points are the same.
#include "common.cuh"
#include <cuda_bf16.h>

namespace b200 {

namespace {

constexpr int kQuantThreads = 256;
constexpr int kClipFactors = 7;   // quant.CLIP_GRID
__device__ constexpr float kClipGrid[kClipFactors] = {1.0f, 0.95f, 0.9f, 0.85f, 0.8f, 0.75f, 0.7f};

// Two fp32 values in one 64-bit register: the packed forms do two multiplications or additions per issue slot.
struct f2 { unsigned long long v; };
DEVI f2 pack2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
DEVI float lo2(f2 a) { return __uint_as_float((uint32_t)a.v); }
DEVI float hi2(f2 a) { return __uint_as_float((uint32_t)(a.v >> 32)); }
DEVI f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
DEVI f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}

DEVI f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// minimum and maximum that keep a NaN (fminf and fmaxf drop it): a damaged weight makes its group's parameters NaN, as torch's
// amin, amax and clamp do, instead of ordinary ones that hide it
DEVI float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
DEVI float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

struct GroupScale { float s, z, rs; };   // scale, zero point, fl(1 / scale)

// scale and zero point of a group with range [lo, hi]
DEVI GroupScale scale_zero(float lo, float hi) {
  GroupScale g;
  const float c15 = 1.0f / 15.0f;
  g.s = __half2float(__float2half_rn(max_nan(__fmul_rn(__fsub_rn(hi, lo), c15), 1e-6f)));
  g.z = min_nan(max_nan(rintf(__fdiv_rn(-lo, g.s)), 0.f), 15.f);
  g.rs = __frcp_rn(g.s);
  return g;
}

// rint(fl(w / s)) of V weights, |w| <= wmax. The product with 1 / s decides unless one of them lies so close to a tie that
// the product's error (1.5 ulp at most) could matter; then all of them are divided. Adding and subtracting 1.5 * 2^23
// rounds half to even for |p| < 2^22 (larger ones fail the test: the margin is then negative); rintf would run at a
// quarter of the rate. The sign bits of (margin - distance) are collected instead of comparing one by one.
template <int V>
DEVI void round_quotients(const float (&w)[V], const GroupScale& g, float wmax, float (&r)[V]) {
  constexpr float kMagic = 12582912.f;
  const float margin = 0.5f - wmax * g.rs * 0x1p-21f;
  const f2 rs2 = pack2(g.rs, g.rs), m2 = pack2(kMagic, kMagic), nm2 = pack2(-kMagic, -kMagic), neg = pack2(-1.f, -1.f);
  uint32_t near = 0;
#pragma unroll
  for (int i = 0; i < V; i += 2) {
    const f2 p = mul2(pack2(w[i], w[i + 1]), rs2), q = add2(add2(p, m2), nm2), d = fma2(q, neg, p);
    r[i] = lo2(q);
    r[i + 1] = hi2(q);
    near |= __float_as_uint(margin - fabsf(lo2(d))) | __float_as_uint(margin - fabsf(hi2(d)));
  }
  if (near >> 31) {
#pragma unroll
    for (int i = 0; i < V; ++i) r[i] = rintf(__fdiv_rn(w[i], g.s));
  }
}

// Sum of the squared rounding errors of V weights: fours first, then the fours. r holds the rounded quotients;
// clamp(r + z, 0, 15) - z = clamp(r, -z, 15 - z): all integers.
template <int V>
DEVI float sum_sq_errors(const float (&w)[V], const float (&r)[V], const GroupScale& g) {
  const f2 s2 = pack2(g.s, g.s);
  const float top = 15.f - g.z;
  float e[V];
#pragma unroll
  for (int i = 0; i < V; i += 2) {
    const f2 c = pack2(fminf(fmaxf(r[i], -g.z), top), fminf(fmaxf(r[i + 1], -g.z), top));
    const f2 d = add2(mul2(c, s2), pack2(-w[i], -w[i + 1])), q = mul2(d, d);
    e[i] = lo2(q);
    e[i + 1] = hi2(q);
  }
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < V; i += 4) {
    const float f = __fadd_rn(__fadd_rn(__fadd_rn(e[i], e[i + 1]), e[i + 2]), e[i + 3]);
    t = i == 0 ? f : __fadd_rn(t, f);
  }
  return t;
}

// `lanes` neighbouring lanes (a power of two) hold one group, V values each; every one of them gets the group's
// parameters and its largest magnitude. With clipping and eight lanes or more, lane f of the group works the parameters of
// factor f out (two divisions, two conversions) and hands them round.
template <int V>
DEVI GroupScale group_params(const float (&w)[V], int lanes, bool clip, float* wmax) {
  float lo = w[0], hi = w[0];
#pragma unroll
  for (int i = 1; i < V; ++i) lo = min_nan(lo, w[i]), hi = max_nan(hi, w[i]);
  for (int o = 1; o < lanes; o <<= 1) {
    lo = min_nan(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = max_nan(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  *wmax = fmaxf(-lo, hi);
  if (!clip) return scale_zero(lo, hi);
  const int lane = threadIdx.x & 31, sub = lane & (lanes - 1);
  const bool shared = lanes >= 8;
  GroupScale own = {0.f, 0.f, 0.f};
  if (shared) {
    const float a = kClipGrid[min(sub, kClipFactors - 1)];
    own = scale_zero(__fmul_rn(lo, a), __fmul_rn(hi, a));
  }
  GroupScale best = own;
  float best_err = 0.f;
#pragma unroll 1
  for (int f = 0; f < kClipFactors; ++f) {
    GroupScale g;
    if (shared) {
      const int src = lane - sub + f;
      g.s = __shfl_sync(0xffffffffu, own.s, src);
      g.z = __shfl_sync(0xffffffffu, own.z, src);
      g.rs = __shfl_sync(0xffffffffu, own.rs, src);
    } else {
      g = scale_zero(__fmul_rn(lo, kClipGrid[f]), __fmul_rn(hi, kClipGrid[f]));
    }
    float r[V];
    round_quotients(w, g, *wmax, r);
    float err = sum_sq_errors(w, r, g);
    for (int o = 1; o < lanes; o <<= 1) err = __fadd_rn(err, __shfl_xor_sync(0xffffffffu, err, o));
    if (f == 0 || err < best_err) best_err = err, best = g;
  }
  return best;
}

template <typename T> DEVI void load8(const T* p, float (&w)[8]);
template <> DEVI void load8<half>(const half* p, float (&w)[8]) { unpack8(*reinterpret_cast<const uint4*>(p), w); }
template <> DEVI void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&w)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) w[2 * i] = __uint_as_float(u[i] << 16), w[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u);
}
template <> DEVI void load8<float>(const float* p, float (&w)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w; w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}

// One thread = 8 consecutive weights = one packed word; G / 8 lanes share a group.
template <typename T>
__global__ void __launch_bounds__(kQuantThreads)
quantize_w4_kernel(const T* __restrict__ W, long long words, int lanes, int clip, const QuantOut out) {
  const long long i = (long long)blockIdx.x * kQuantThreads + threadIdx.x;
  const bool live = i < words;   // groups are whole: the lanes of a group are live together
  float w[8];
  load8(W + 8 * (live ? i : words - 1), w);
  float wmax;
  const GroupScale g = group_params<8>(w, lanes, clip, &wmax);
  if (!live) return;
  float lv[8];
  uint32_t q[8];
  round_quotients(w, g, wmax, lv);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    lv[e] = fminf(fmaxf(__fadd_rn(lv[e], g.z), 0.f), 15.f);
    q[e] = (uint32_t)lv[e];
  }
  if (out.packed) {
    uint32_t p = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) p |= q[e] << (4 * (e >> 1) + 16 * (e & 1));
    out.packed[i] = p;
  }
  if (out.q)
    out.q[i] = make_uint2(q[0] | q[1] << 8 | q[2] << 16 | q[3] << 24, q[4] | q[5] << 8 | q[6] << 16 | q[7] << 24);
  if (out.deq) {
    uint32_t h[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      h[e] = as_u32(__floats2half2_rn(__fmul_rn(lv[2 * e] - g.z, g.s), __fmul_rn(lv[2 * e + 1] - g.z, g.s)));
    out.deq[i] = make_uint4(h[0], h[1], h[2], h[3]);
  }
  if ((threadIdx.x & (lanes - 1)) == 0) {
    const long long gi = i / lanes;
    if (out.sz) out.sz[gi] = __floats2half2_rn(g.s, g.z);
    if (out.scale) out.scale[gi] = __float2half_rn(g.s), out.zero[gi] = __float2half_rn(g.z);
  }
}

constexpr int kGptqWarps = 8, kGptqBlock = 128;   // rows per CTA; columns of a block, four per lane

// W fp32 [N, ldw]: columns [0, nb) of it are the block (already updated by the blocks to its left). U: the block's nb x nb
// part of the upper factor, element (i, j) at U[i * us0 + j * us1]. Q, S, Z point at the block's first column / group.
__global__ void __launch_bounds__(kGptqWarps * 32)
gptq_block_kernel(const float* __restrict__ W, int ldw, int N, int nb, const float* __restrict__ U, long long us0,
                  long long us1, int group, int clip, uint8_t* __restrict__ Q, int ldq, float* __restrict__ S,
                  float* __restrict__ Z, int lds, float* __restrict__ E, int lde) {
  extern __shared__ __align__(16) float u_s[];   // [nb][kGptqBlock], zero beyond nb
  const int tid = threadIdx.x, lane = tid & 31, row = blockIdx.x * kGptqWarps + (tid >> 5);
  for (int k = tid; k < nb * kGptqBlock; k += kGptqWarps * 32) {
    // consecutive threads walk the direction that is contiguous in memory
    const int i = us1 == 1 ? k / kGptqBlock : k % nb, j = us1 == 1 ? k % kGptqBlock : k / nb;
    u_s[i * kGptqBlock + j] = j < nb ? U[i * us0 + j * us1] : 0.f;
  }
  __syncthreads();
  if (row >= N) return;
  const int c0 = 4 * lane;
  const bool mine = c0 < nb;   // nb is a multiple of four
  float w[4] = {0.f, 0.f, 0.f, 0.f}, err[4] = {0.f, 0.f, 0.f, 0.f};
  if (mine) {
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] = W[(size_t)row * ldw + c0 + k];
  }
  uint32_t levels = 0;
  GroupScale g = {1.f, 0.f, 1.f};
  for (int ol = 0; 4 * ol < nb; ++ol) {   // lane `ol` owns columns 4 ol .. 4 ol + 3
    if ((4 * ol) % group == 0) {          // a group starts: its range from the weights as they are now
      float wmax;
      g = group_params<4>(w, group >> 2, clip, &wmax);
      g.s = __shfl_sync(0xffffffffu, g.s, ol);
      g.z = __shfl_sync(0xffffffffu, g.z, ol);
      g.rs = __shfl_sync(0xffffffffu, g.rs, ol);
      if (lane == ol) S[(size_t)row * lds + 4 * ol / group] = g.s, Z[(size_t)row * lds + 4 * ol / group] = g.z;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = 4 * ol + k;
      const float col = __shfl_sync(0xffffffffu, w[k], ol);
      const float two[2] = {col, 0.f};
      float r[2];
      round_quotients(two, g, fabsf(col), r);
      const float lv = fminf(fmaxf(__fadd_rn(r[0], g.z), 0.f), 15.f);
      const float4 u = *reinterpret_cast<const float4*>(u_s + i * kGptqBlock + c0);
      const float e = __fdiv_rn(__fsub_rn(col, __fmul_rn(lv - g.z, g.s)), u_s[i * kGptqBlock + i]);
      // columns at or before i are not read again, so they may take part
      w[0] = __fsub_rn(w[0], __fmul_rn(e, u.x));
      w[1] = __fsub_rn(w[1], __fmul_rn(e, u.y));
      w[2] = __fsub_rn(w[2], __fmul_rn(e, u.z));
      w[3] = __fsub_rn(w[3], __fmul_rn(e, u.w));
      if (lane == ol) levels |= (uint32_t)lv << (8 * k), err[k] = e;
    }
  }
  if (mine) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      Q[(size_t)row * ldq + c0 + k] = (uint8_t)(levels >> (8 * k));
      E[(size_t)row * lde + c0 + k] = err[k];
    }
  }
}

}  // namespace

// dtype: 0 fp16, 1 bf16, 2 fp32. G: a power of two, 8 .. 256, that divides K.
cudaError_t quantize_w4_dispatch(const void* W, int dtype, int N, int K, int G, int clip, const QuantOut& out,
                                 cudaStream_t st) {
  const long long words = (long long)N * K / 8;
  const unsigned blocks = (unsigned)((words + kQuantThreads - 1) / kQuantThreads);
  if (dtype == 0) quantize_w4_kernel<half><<<blocks, kQuantThreads, 0, st>>>((const half*)W, words, G / 8, clip, out);
  else if (dtype == 1)
    quantize_w4_kernel<__nv_bfloat16><<<blocks, kQuantThreads, 0, st>>>((const __nv_bfloat16*)W, words, G / 8, clip, out);
  else quantize_w4_kernel<float><<<blocks, kQuantThreads, 0, st>>>((const float*)W, words, G / 8, clip, out);
  return cudaPeekAtLastError();
}

cudaError_t gptq_block_dispatch(const float* W, int ldw, int N, int nb, const float* U, long long us0, long long us1,
                                int group, int clip, uint8_t* Q, int ldq, float* S, float* Z, int lds, float* E, int lde,
                                cudaStream_t st) {
  const size_t smem = (size_t)nb * kGptqBlock * sizeof(float);
  static size_t allowed[kMaxDevices] = {};
  const cudaError_t e = allow_dynamic_smem(gptq_block_kernel, smem, allowed);
  if (e != cudaSuccess) return e;
  gptq_block_kernel<<<(N + kGptqWarps - 1) / kGptqWarps, kGptqWarps * 32, smem, st>>>(
      W, ldw, N, nb, U, us0, us1, group, clip, Q, ldq, S, Z, lds, E, lde);
  return cudaPeekAtLastError();
}

}  // namespace b200
