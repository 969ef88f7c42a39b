// Attention of a prompt: T query tokens at positions start .. start + T - 1 over one sequence's paged cache (their own keys and
// values already appended), causal, grouped-query heads.
//
// A CTA owns 128 query rows of one kv head - row = (token, head of the group), so the heads of a group share what is read - and
// walks over the context in tiles of 64 tokens with an online softmax (FlashAttention, Dao et al. 2022) on the 5th-generation tensor
// cores: S = Q K^T and O += P V are tcgen05.mma with accumulators in tensor memory; a softmax thread owns one row of S, and its
// probabilities go back to tensor memory as the A operand of the second product. Per tile and row the thread does 64 exponentials, at
// 16 a clock and SM: that, 61 us for 4096 tokens x 32 heads, is the floor here, so everything else runs beside it - S and P have two
// buffers each, one warp issues the MMAs of the next tile meanwhile, two warps copy cached rows (cp.async, into the 128-byte-swizzled
// layout), and at head_dim 64 two CTAs share an SM. The running maximum follows with a delay: O is rescaled only when the maximum has
// grown by more than 2^8 (Zadouri et al., FlashAttention-4), which fp16 probabilities and fp32 sums take without loss.
//   4096 tokens, 32 heads on 4 kv heads x 64: 143 us (277 with warp-level MMAs; the decode kernel, one pass over the cache per query
//   token, took 1.8 ms). 512 tokens: 15.7 us (15.5 and 19.3 for the merge of its splits).
// Where a short prompt continues a long context the CTAs are few: up to 8 CTAs (a cluster) then share the context of a row block and
// merge through distributed shared memory.
// Warps: 0-3 softmax (warp q owns rows 32 q ..), 4 MMA issue, 5-6 loads. Tensor memory columns: S 2 x 64, P 2 x 32, O head_dim.
// Every wait is bounded; a wait that runs out raises the CTA's fail flag, all roles leave, the CTA waits (bounded) for its MMAs, joins
// the cluster barriers, frees its tensor memory, and b200_gemm_w4a16_status is non-zero.
#include "prefill.h"
#include "umma.cuh"
#include <math_constants.h>

namespace b200 {

namespace {

using namespace umma;

__device__ int g_prefill_attn_status = 0;   // 0, or the code of the first wait that ran out

constexpr int kRows = 128, kTile = 64, kStages = 4, kLag = 1, kMaxSplit = 8;
constexpr int kSoftWarps = 4, kMmaWarp = 4, kLoadWarps = 2, kThreads = (kSoftWarps + 1 + kLoadWarps) * 32;
constexpr float kGrow = 8.f;   // base-2 growth of the maximum that is let pass
enum : int { WAIT_KV = 17, WAIT_S_FREE = 18, WAIT_P = 19, WAIT_S = 20, WAIT_PV = 21, WAIT_STAGE = 22 };

template <int D> constexpr int stage_bytes() { return 2 * kTile * D * 2; }   // K rows then V rows
template <int D> constexpr size_t smem_bytes() { return 1024 + (size_t)kRows * D * 2 + (size_t)kStages * stage_bytes<D>(); }
template <int D> constexpr int tmem_columns() { return D == 64 ? 256 : 512; }

struct Shared {
  uint64_t kv_full[kStages], kv_empty[kStages], s_full[2], s_empty[2], p_full[2], pv_done[2], drain;
  uint32_t tmem;
  int fail;
};

DEVI float ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
DEVI float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// byte offset of 16-byte piece p (of a row of 64-wide blocks of `rows` rows) of row r in the swizzled layout
DEVI uint32_t swz_piece(int r, int p, int rows) { return (uint32_t)((p >> 3) * rows * 128 + r * 128 + (((p & 7) ^ (r & 7)) << 4)); }

// the elected lane's MMAs so far -> one arrival on bar (whole warp)
DEVI void commit(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(sa(bar))
      : "memory");
}
// D (+)= A B with A in shared memory / in tensor memory; issued by the elected lane (whole warp)
DEVI void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred e, p;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
DEVI void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred e, p;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

}  // namespace

// Grid (row blocks, n_kv, splits), clusters (1, 1, splits). q rows: token t at q + t * q_stride, heads one after the other. PS tokens of
// context per split (a multiple of kTile).
template <int D>
__global__ void __launch_bounds__(kThreads, D == 64 ? 2 : 1)
prefill_attn_kernel(const half* __restrict__ q, int q_stride, const half* __restrict__ kc, const half* __restrict__ vc,
                    const int* __restrict__ bt, int start, int T, int n_kv, int log2hpg, int log2P, int PS, float sl2,
                    half* __restrict__ out) {
  constexpr int PP = D / 8, CHUNKS = D / 64, STAGE = stage_bytes<D>();
  constexpr uint32_t kP = 2 * kTile, kO = 3 * kTile;   // tensor-memory columns of P and O
  extern __shared__ uint8_t raw[];
  __shared__ Shared sh;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = base + kRows * D * 2;   // behind Q
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int hpg = 1 << log2hpg, n_q = n_kv << log2hpg, C = gridDim.z;
  const int rb = gridDim.x - 1 - blockIdx.x;   // late tokens see the most context: they start first
  const int kvh = blockIdx.y, split = blockIdx.z, row0 = rb * kRows;
  const int last = start + min(T - 1, (row0 + kRows - 1) >> log2hpg);   // the block's last position
  const int k0 = split * PS, k1 = min(last + 1, k0 + PS);
  const int ntiles = k0 < k1 ? (k1 - k0 + kTile - 1) / kTile : 0;
  volatile int* fail = &sh.fail;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(&sh.tmem)), "n"(tmem_columns<D>()) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) bar_init(&sh.kv_full[i], kLoadWarps), bar_init(&sh.kv_empty[i], 1);
    for (int i = 0; i < 2; ++i)
      bar_init(&sh.s_full[i], 1), bar_init(&sh.s_empty[i], kSoftWarps), bar_init(&sh.p_full[i], kSoftWarps), bar_init(&sh.pv_done[i], 1);
    bar_init(&sh.drain, 1);
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pdl_wait();
  // Q: rows of 128 bytes per 64 dims, swizzled
  for (int i = tid; i < kRows * PP; i += kThreads) {
    const int r = i / PP, p = i % PP, t = min((row0 + r) >> log2hpg, T - 1), h = (kvh << log2hpg) + ((row0 + r) & (hpg - 1));
    *reinterpret_cast<uint4*>(base + swz_piece(r, p, kRows)) = *reinterpret_cast<const uint4*>(q + (size_t)t * q_stride + (size_t)h * D + 8 * p);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch_dependents();   // with this CTA's tensor memory allocated (see prefill_gemm_tiled_kernel)
  const uint32_t tmem = sh.tmem;

  float m = -CUDART_INF_F, l = 0.f;   // softmax thread: reference maximum (base-2 units) and sum of its row
  if (warp < kSoftWarps) {
    const uint32_t tq = tmem + ((uint32_t)(32 * warp) << 16);
    const int r = row0 + tid, pos = start + min(r >> log2hpg, T - 1);
    const int wfirst = start + min(T - 1, (row0 + 32 * warp) >> log2hpg);   // the warp's first position
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < ntiles; ++i) {
      const int b = i & 1;
      ok = __all_sync(0xffffffffu, bar_wait<0>(&sh.s_full[b], (i >> 1) & 1, fail, &g_prefill_attn_status, WAIT_S));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[kTile];
#pragma unroll
      for (int c = 0; c < kTile; c += 16) tmem_ld16_async(tq + (uint32_t)(kTile * b + c), s + c);
      tmem_wait_ld(s);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&sh.s_empty[b]);
      const int j0 = k0 + i * kTile;
      if (j0 + kTile - 1 > wfirst) {   // the diagonal runs through this tile
        const int seen = pos - j0;
#pragma unroll
        for (int c = 0; c < kTile; ++c)
          if (c > seen) s[c] = -CUDART_INF_F;
      }
      float mx = fmaxf(s[0], s[1]);
#pragma unroll
      for (int c = 2; c < kTile; c += 2) mx = max3(mx, s[c], s[c + 1]);
      mx *= sl2;
      const bool grow = mx > m + kGrow || (m == -CUDART_INF_F && mx > m);
      if (__any_sync(0xffffffffu, grow)) {
        const float f = grow ? ex2(m - mx) : 1.f;   // m = -inf: 0
        if (grow) m = mx;
        l *= f;
        if (i > 0) {   // O as of tile i - 1
          ok = __all_sync(0xffffffffu, bar_wait<0>(&sh.pv_done[b ^ 1], ((i - 1) >> 1) & 1, fail, &g_prefill_attn_status, WAIT_PV));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c = 0; c < D; c += 16) {
            uint32_t o[16];
            tmem_ld16(tq + kO + c, o);
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
            tmem_st16(tq + kO + c, o);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
      }
      const float sub = m == -CUDART_INF_F ? 0.f : m;   // nothing visible yet: every probability is 2^-inf
      uint32_t p[kTile / 2];
      float l0 = 0.f, l1 = 0.f;
#pragma unroll
      for (int c = 0; c < kTile; c += 2) {
        const float x = ex2(fmaf(s[c], sl2, -sub)), y = ex2(fmaf(s[c + 1], sl2, -sub));
        l0 += x;
        l1 += y;
        p[c / 2] = as_u32(__floats2half2_rn(x, y));
      }
      l += l0 + l1;
      if (i >= 2) {
        ok = __all_sync(0xffffffffu, bar_wait<0>(&sh.pv_done[b], ((i - 2) >> 1) & 1, fail, &g_prefill_attn_status, WAIT_PV));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
#pragma unroll
      for (int c = 0; c < kTile / 2; c += 16) tmem_st16(tq + kP + (uint32_t)(kTile / 2 * b + c), p + c);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&sh.p_full[b]);
    }
    if (ok && ntiles > 0) {   // the last product
      const int i = ntiles - 1;
      __all_sync(0xffffffffu, bar_wait<0>(&sh.pv_done[i & 1], (i >> 1) & 1, fail, &g_prefill_attn_status, WAIT_PV));
    }
  } else if (warp == kMmaWarp) {
    // M = 128; S: N = 64, both operands K-major; O: N = D, B (V) MN-major (bit 16)
    constexpr uint32_t idesc_s = (1u << 4) | ((kTile >> 3) << 17) | ((128u >> 4) << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (1u << 16) | ((D >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t q_s = sa(base), ring_s = sa(ring);
    auto scores = [&](int i) {   // S of tile i
      const uint32_t k_s = ring_s + (i % kStages) * STAGE;
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
        mma_ss(tmem + (uint32_t)(kTile * (i & 1)), desc_sw128(q_s + (k / 4) * (kRows * 128)) + 2 * (k % 4),
               desc_sw128(k_s + (k / 4) * (kTile * 128)) + 2 * (k % 4), idesc_s, k > 0);
      commit(&sh.s_full[i & 1]);
    };
    auto arrived = [&](uint64_t* bar, uint32_t parity, int code) {
      const bool ok = __all_sync(0xffffffffu, bar_wait<0>(bar, parity, fail, &g_prefill_attn_status, code));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    bool ok = ntiles > 0 && arrived(&sh.kv_full[0], 0, WAIT_KV);
    if (ok) scores(0);
#pragma unroll 1
    for (int i = 0; i < ntiles && ok; ++i) {
      const int n = i + 1;
      if (n < ntiles) {
        ok = arrived(&sh.kv_full[n % kStages], (n / kStages) & 1, WAIT_KV) &&
             (n < 2 || arrived(&sh.s_empty[n & 1], ((n - 2) >> 1) & 1, WAIT_S_FREE));
        if (!ok) break;
        scores(n);
      }
      ok = arrived(&sh.p_full[i & 1], (i >> 1) & 1, WAIT_P);
      if (!ok) break;
      const uint32_t v_s = ring_s + (i % kStages) * STAGE + kTile * D * 2;
#pragma unroll
      for (int k = 0; k < kTile / 16; ++k)
        mma_ts(tmem + kO, tmem + kP + (uint32_t)(kTile / 2 * (i & 1) + 8 * k), desc_sw128(v_s, kTile * 128) + 128 * k, idesc_o, i > 0 || k > 0);
      commit(&sh.pv_done[i & 1]);
      commit(&sh.kv_empty[i % kStages]);
    }
    commit(&sh.drain);   // whatever was issued has completed before the CTA's memory goes away
    for (int i = 0; i < (1 << 16) && !bar_try(&sh.drain, 0); ++i) __nanosleep(32);
  } else {
    const int lt = tid - 32 * (kSoftWarps + 1);
    bool ok = true;
    auto hand_over = [&](int i) {   // this warp's pieces of tile i have landed
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&sh.kv_full[i % kStages]);
    };
#pragma unroll 1
    for (int i = 0; i < ntiles; ++i) {
      if (i >= kStages) {
        ok = __all_sync(0xffffffffu, bar_wait<32>(&sh.kv_empty[i % kStages], (i / kStages - 1) & 1, fail, &g_prefill_attn_status, WAIT_STAGE));
        if (!ok) break;
      }
      const uint32_t k_s = sa(ring) + (i % kStages) * STAGE;
      constexpr int RPI = kLoadWarps * 32 / PP;   // rows per iteration
#pragma unroll 8
      for (int k = 0; k < kTile / RPI; ++k) {
        const int r = lt / PP + RPI * k, p = lt % PP, j = min(k0 + i * kTile + r, last);   // past the context: its last token again (masked)
        const size_t off = ((((size_t)__ldg(bt + (j >> log2P)) * n_kv + kvh) << log2P) + (j & ((1 << log2P) - 1))) * D + 8 * p;
        const uint32_t to = k_s + swz_piece(r, p, kTile);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(kc + off) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + kTile * D * 2), "l"(vc + off) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (i >= kLag) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kLag) : "memory");
        hand_over(i - kLag);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (ok)
      for (int i = max(0, ntiles - kLag); i < ntiles; ++i) hand_over(i);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  constexpr int OP = D + 4;   // floats per row of a parked partial: 16-byte stores by 32 rows at once hit all banks
  float* park = reinterpret_cast<float*>(ring);               // [kRows][OP], over the idle stages
  float2* ml = reinterpret_cast<float2*>(park + kRows * OP);  // [kRows]
  static_assert(kRows * OP * 4 + kRows * 8 <= kStages * STAGE, "partials fit over the stages");
  if (warp < kSoftWarps && !*fail) {
    const int r = row0 + tid, t = r >> log2hpg, h = (kvh << log2hpg) + (r & (hpg - 1));
    const uint32_t tq = tmem + ((uint32_t)(32 * warp) << 16) + kO;
    const float f = C == 1 ? 1.f / l : 1.f;
    half* o = out + ((size_t)t * n_q + h) * D;
#pragma unroll 1
    for (int c = 0; c < D; c += 16) {
      uint32_t v[16];
      if (ntiles > 0) {
        tmem_ld16(tq + c, v);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0u;
      }
      if (C == 1) {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = as_u32(__floats2half2_rn(__uint_as_float(v[2 * e]) * f, __uint_as_float(v[2 * e + 1]) * f));
        if (t < T) {
          reinterpret_cast<uint4*>(o + c)[0] = make_uint4(w[0], w[1], w[2], w[3]);
          reinterpret_cast<uint4*>(o + c)[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 16; e += 4)
          *reinterpret_cast<uint4*>(park + tid * OP + c + e) = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      }
    }
    ml[tid] = make_float2(m, l);
  }
  if (C > 1) {
    cluster_barrier();
    if (!*fail) {   // CTA `split` finishes every C-th row; a thread takes four dims
      for (int i = tid; i < kRows / C * (D / 4); i += kThreads) {
        const int rr = (i / (D / 4)) * C + split, d = 4 * (i % (D / 4)), r = row0 + rr, t = r >> log2hpg;
        const uint32_t at = sa(park + rr * OP + d), am = sa(ml + rr);
        float mm[kMaxSplit], ll[kMaxSplit], M = -CUDART_INF_F, L = 0.f;
        float4 v[kMaxSplit], o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int c = 0; c < kMaxSplit; ++c) {
          mm[c] = -CUDART_INF_F;
          if (c < C) {
            v[c] = ld_cluster4(in_cta(at, c));
            asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(mm[c]), "=f"(ll[c]) : "r"(in_cta(am, c)) : "memory");
          }
        }
#pragma unroll
        for (int c = 0; c < kMaxSplit; ++c) M = fmaxf(M, mm[c]);   // finite: position 0 is in split 0
#pragma unroll
        for (int c = 0; c < kMaxSplit; ++c)
          if (c < C) {
            const float a = ex2(mm[c] - M);
            L = fmaf(a, ll[c], L);
            o.x = fmaf(a, v[c].x, o.x), o.y = fmaf(a, v[c].y, o.y), o.z = fmaf(a, v[c].z, o.z), o.w = fmaf(a, v[c].w, o.w);
          }
        const float f = 1.f / L;
        if (t < T)
          *reinterpret_cast<uint2*>(out + ((size_t)t * n_q + (kvh << log2hpg) + (r & (hpg - 1))) * D + d) =
              make_uint2(as_u32(__floats2half2_rn(o.x * f, o.y * f)), as_u32(__floats2half2_rn(o.z * f, o.w * f)));
      }
    }
    cluster_barrier();   // nobody's shared memory goes away while a peer still reads it
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(tmem_columns<D>()) : "memory");
}

bool prefill_attention_takes(int D, int n_q, int n_kv) {
  const int hpg = n_q / n_kv;
  return (D == 64 || D == 128) && (hpg & (hpg - 1)) == 0 && hpg <= kRows;
}

cudaError_t prefill_attention_status(int* code) {
  return cudaMemcpyFromSymbol(code, g_prefill_attn_status, sizeof(int), 0, cudaMemcpyDeviceToHost);
}

cudaError_t prefill_attention_dispatch(const void* q, int q_stride, const void* kc, const void* vc, const int* bt, int start, int T,
                                       int n_q, int n_kv, int D, int log2P, void* out, cudaStream_t st) {
  const int hpg = n_q / n_kv;
  int log2hpg = 0;
  while ((1 << log2hpg) < hpg) ++log2hpg;
  const int row_blocks = (T * hpg + kRows - 1) / kRows, tiles = (start + T + kTile - 1) / kTile;
  // one wave of CTAs (two an SM at head_dim 64), four tiles each at least so that a split outweighs its merge (~2 us)
  const int slots = kNumSMs * (D == 64 ? 2 : 1);
  int C = 1;
  while (C < kMaxSplit && row_blocks * n_kv * C * 2 <= slots && tiles >= 4 * 2 * C) C *= 2;
  const int PS = (tiles + C - 1) / C * kTile;
  auto kern = D == 64 ? prefill_attn_kernel<64> : prefill_attn_kernel<128>;
  const size_t smem = D == 64 ? smem_bytes<64>() : smem_bytes<128>();
  static size_t allowed[2][kMaxDevices] = {};
  const cudaError_t e = allow_dynamic_smem(kern, smem, allowed[D == 128]);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = C;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(row_blocks, n_kv, C);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, (const half*)q, q_stride, (const half*)kc, (const half*)vc, bt, start, T, n_kv, log2hpg, log2P,
                            PS, 1.44269504088896340736f / sqrtf((float)D), (half*)out);
}

}  // namespace b200
