// Attention of a prompt: T query tokens at positions start .. start + T - 1 over one sequence's paged cache (their own keys and
// values already appended), causal, grouped-query heads.
//
// A CTA owns 128 query rows of one kv head - row = (token, head of the group), so the heads of a group share what is read - and
// walks over the context in tiles of 64 tokens with an online softmax (FlashAttention, Dao et al. 2022) on the 5th-generation tensor
// cores: S = Q K^T and O += P V are tcgen05.mma with accumulators in tensor memory; a softmax thread owns one row of S and puts its
// probabilities back over the scores, as the A operand of the second product. Per tile and row the thread does 64 exponentials, at
// 16 a clock and SM: that, 61 us for 4096 tokens x 32 heads, is the floor here, so everything else runs beside it: the scores have two
// buffers, so that those of the next tile are there when a tile is done; one warp issues the MMAs; half the loading warps copy cached
// rows of K, half of V (cp.async, into the 128-byte-swizzled layout); two CTAs share an SM. The running maximum follows with a delay:
// O is rescaled only when the maximum has grown by more than 2^8 (Zadouri et al., FlashAttention-4). Against such a maximum no
// probability of a row is exactly 1, so fp16 alone would lose what the exact maximum keeps: the probabilities enter the second product
// twice, as fp16 value and as fp16 remainder. Error against 64 bits, 200 tokens behind 1800: 2.08e-4, which is the rounding of the
// output (2.88e-4 with the values alone; 2.52e-4 in fp16 against the exact maximum). It costs 23 of the 129 us at 4096 tokens.
//   4096 tokens, 32 heads on 4 kv heads x 64: 129 us (277 with warp-level MMAs; the decode kernel, one pass over the cache per query
//   token, took 1.8 ms). 512 tokens: 11 us.
// What it waited for on the way, at 4096 tokens and without the remainders: 127 us with K and V in one ring whose loaders handed a tile over late; 119 with two
// groups of softmax warps that take turns (scores of the next tile then come only behind the product of this one); queries through
// registers, one round trip after the other, cost 3 us a CTA.
// Where a short prompt continues a long context the CTAs are few: up to 8 CTAs (a cluster) then share the context of a row block and
// merge through distributed shared memory.
// Warps: 0-3 softmax (warp q owns rows 32 q ..), 4 MMA issue, from 5 loads. Tensor memory columns: S and P 2 x 64, O head_dim.
// Every wait is bounded; a wait that runs out raises the CTA's fail flag, all roles leave, the CTA waits (bounded) for its MMAs, joins
// the cluster barriers, frees its tensor memory, and b200_gemm_w4a16_status is non-zero.
#include "prefill.h"
#include "umma.cuh"
#include <math_constants.h>

namespace b200 {

namespace {

using namespace umma;

__device__ int g_prefill_attn_status = 0;   // 0, or the code of the first wait that ran out

constexpr int kRows = 128, kTile = 64, kMaxSplit = 8;
constexpr int kSoftWarps = 4, kMmaWarp = kSoftWarps, kMaxStages = 5;
constexpr float kGrow = 8.f;   // base-2 growth of the maximum that is let pass
enum : int { WAIT_K = 17, WAIT_V = 18, WAIT_P = 19, WAIT_S = 20, WAIT_PV = 21, WAIT_STAGE = 22, WAIT_Q = 23, WAIT_DRAIN = 24 };

template <int D> constexpr int load_warps() { return D / 32; }
template <int D> constexpr int threads() { return (kMmaWarp + 1 + load_warps<D>()) * 32; }
template <int D> constexpr int tile_bytes() { return kTile * D * 2; }   // of K or of V
template <int D> constexpr int stages() { return D == 64 ? 5 : 2; }     // tiles of K, and as many of V
template <int D> constexpr size_t smem_bytes() { return 1024 + (size_t)kRows * D * 2 + (size_t)2 * stages<D>() * tile_bytes<D>(); }
constexpr int kTmemColumns = 256;   // two CTAs an SM

struct Shared {
  uint64_t k_full[kMaxStages], k_empty[kMaxStages], v_full[kMaxStages], v_empty[kMaxStages], s_full[2], p_full[2], pv_done[2], q_full, drain;
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
// two floats in one register pair
DEVI uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
DEVI void unpair(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
DEVI uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
DEVI uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
DEVI uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
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

// A token must not depend on later ones, but the products above multiply whole tiles: a probability of zero against an infinity or a
// NaN in the value row of a later token of the block is NaN. Where that may be why some of the dims [d0, d1) of a row came out NaN, they
// are computed once more from the tokens the row sees, by one thread (a row that sees a NaN itself stays as it is). Kept out of
// line, behind one test per row: the code of it in the epilogue costs a short prompt 1 us a launch.
struct RowArgs {
  const half *q, *kc, *vc;   // the row's query; the caches
  const int* bt;
  int kvh, n_kv, log2P, pos, last;   // last: the last position the row was multiplied with
  float sl2;
  half* out;                 // the row
};
template <int D>
__device__ __noinline__ void redo_row(const RowArgs a, int d0, int d1) {
  auto row = [&](int j) { return (((((size_t)a.bt[j >> a.log2P] * a.n_kv + a.kvh) << a.log2P) + (j & ((1 << a.log2P) - 1))) * D); };
#pragma unroll 1
  for (int d = d0; d < d1; d += 4) {
    const uint2 was = *reinterpret_cast<const uint2*>(a.out + d);
    const half2 z = __hadd2(as_h2(was.x), as_h2(was.y));
    if (!__hisnan(__low2half(z)) && !__hisnan(__high2half(z))) continue;
    bool hidden = false;
#pragma unroll 1
    for (int j = a.pos + 1; j <= a.last; ++j) {
      const uint2 v = *reinterpret_cast<const uint2*>(a.vc + row(j) + d);
      hidden |= (v.x & 0x7C00u) == 0x7C00u || (v.x & 0x7C000000u) == 0x7C000000u || (v.y & 0x7C00u) == 0x7C00u || (v.y & 0x7C000000u) == 0x7C000000u;
    }
    if (!hidden) continue;
    float m = -CUDART_INF_F, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int j = 0; j <= a.pos; ++j) {
      const size_t at = row(j);
      float s = 0.f;
#pragma unroll 1
      for (int c = 0; c < D; c += 8) {
        float x[8], y[8];
        unpack8(*reinterpret_cast<const uint4*>(a.q + c), x);
        unpack8(*reinterpret_cast<const uint4*>(a.kc + at + c), y);
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(x[e], y[e], s);
      }
      s *= a.sl2;
      if (s != s) return;
      const float mn = fmaxf(m, s), f = m == mn ? 1.f : exp2f(m - mn), p = s == -CUDART_INF_F ? 0.f : exp2f(s - mn);
      m = mn, l = fmaf(l, f, p);
      const uint2 v = *reinterpret_cast<const uint2*>(a.vc + at + d);
      const float2 v0 = __half22float2(as_h2(v.x)), v1 = __half22float2(as_h2(v.y));
      const float w[4] = {v0.x, v0.y, v1.x, v1.y};
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = fmaf(p, w[e], o[e] * f);
    }
    const float f = 1.f / l;
    *reinterpret_cast<uint2*>(a.out + d) = make_uint2(as_u32(__floats2half2_rn(o[0] * f, o[1] * f)), as_u32(__floats2half2_rn(o[2] * f, o[3] * f)));
  }
}

}  // namespace

// Grid (row blocks x n_kv, 1, splits), clusters (1, 1, splits). q rows: token t at q + t * q_stride, heads one after the other.
template <int D>
__global__ void __launch_bounds__(threads<D>(), 2)
prefill_attn_kernel(const half* __restrict__ q, int q_stride, const half* __restrict__ kc, const half* __restrict__ vc,
                    const int* __restrict__ bt, int start, int T, int n_kv, int log2hpg, int log2P, float sl2,
                    half* __restrict__ out) {
  constexpr int PP = D / 8, TILE = tile_bytes<D>(), NS = stages<D>(), LW = load_warps<D>(), kLag = NS > 2 ? 2 : 1;
  constexpr uint32_t kO = 2 * kTile;   // tensor-memory column of O
  extern __shared__ uint8_t raw[];
  __shared__ Shared sh;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = base + kRows * D * 2;   // behind Q
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int hpg = 1 << log2hpg, n_q = n_kv << log2hpg, C = gridDim.z;
  // late tokens see the most context: they start first, for all kv heads
  const int rb = (gridDim.x - 1 - blockIdx.x) / n_kv, kvh = blockIdx.x % n_kv, split = blockIdx.z, row0 = rb * kRows;
  const int last = start + min(T - 1, (row0 + kRows - 1) >> log2hpg);   // the block's last position
  const int tiles = last / kTile + 1, each = (tiles + C - 1) / C, k0 = split * each * kTile;   // context of this CTA: each tiles from k0
  const int ntiles = max(0, min(each, tiles - split * each));
  volatile int* fail = &sh.fail;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sa(&sh.tmem)), "n"(kTmemColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < NS; ++i) {
      bar_init(&sh.k_full[i], LW / 2), bar_init(&sh.k_empty[i], 1);
      bar_init(&sh.v_full[i], LW / 2), bar_init(&sh.v_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) bar_init(&sh.s_full[i], 1), bar_init(&sh.p_full[i], kSoftWarps), bar_init(&sh.pv_done[i], 1);
    bar_init(&sh.q_full, kSoftWarps), bar_init(&sh.drain, 1);
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  pdl_launch_dependents();   // with this CTA's tensor memory allocated (see prefill_gemm_tiled_kernel)
  const uint32_t tmem = sh.tmem;
  // a loading warp's rows lane and lane + 32 of its first tile: the block table does not come from the kernels before this one, and its
  // round trip would stand in front of every other (embed_rows_kernel lets nothing of a chunk start before what precedes the chunk is done)
  constexpr int RW = kTile / (LW / 2);   // rows of a tile per loading warp
  const int first = ((warp - kMmaWarp - 1) >> 1) * RW;
  auto row = [&](int i, int r) {   // row r of this warp's part of tile i in the cache, in units of D; behind the context: the last (masked)
    const int j = min(k0 + i * kTile + first + r, last);
    return ((__ldg(bt + (j >> log2P)) * n_kv + kvh) << log2P) + (j & ((1 << log2P) - 1));
  };
  int lo = 0, hi = 0;
  if (warp > kMmaWarp && ntiles > 0) lo = row(0, lane), hi = RW > 32 ? row(0, lane + 32) : 0;
  pdl_wait();

  float m = -CUDART_INF_F, l = 0.f;   // softmax thread: reference maximum (base-2 units) and sum of its row
  const uint32_t tq = tmem + ((uint32_t)(32 * warp) << 16);
  if (warp < kSoftWarps) {
    if (ntiles > 0) {   // Q: rows of 128 bytes per 64 dims, swizzled
#pragma unroll
      for (int i = tid; i < kRows * PP; i += kSoftWarps * 32) {
        const int r = i / PP, p = i % PP, t = min((row0 + r) >> log2hpg, T - 1), h = (kvh << log2hpg) + ((row0 + r) & (hpg - 1));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa(base) + swz_piece(r, p, kRows)),
                     "l"(q + (size_t)t * q_stride + (size_t)h * D + 8 * p)
                     : "memory");
      }
      asm volatile("cp.async.wait_all;" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&sh.q_full);
    }
    const int pos = start + min((row0 + tid) >> log2hpg, T - 1);
    const int wfirst = start + min(T - 1, (row0 + 32 * warp) >> log2hpg);   // the warp's first position
    uint64_t sum[2] = {0, 0};   // pairs of partial sums
#pragma unroll 1
    for (int i = 0; i < ntiles; ++i) {
      const int b = i & 1;
      const uint32_t ts = tq + (uint32_t)(kTile * b);
      if (!__all_sync(0xffffffffu, bar_wait<0>(&sh.s_full[b], (i >> 1) & 1, fail, &g_prefill_attn_status, WAIT_S))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float s[kTile];
#pragma unroll
      for (int c = 0; c < kTile; c += 16) tmem_ld16_async(ts + c, s + c);
      tmem_wait_ld(s);
      const int j0 = k0 + i * kTile;
      if (j0 + kTile - 1 > wfirst) {   // the diagonal runs through this tile
        const int seen = pos - j0;
#pragma unroll
        for (int c = 0; c < kTile; ++c)
          if (c > seen) s[c] = -CUDART_INF_F;
      }
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = fmaxf(s[e], s[kTile - 4 + e]);
#pragma unroll
      for (int c = 4; c < kTile - 4; c += 8)
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = max3(x[e], s[c + 2 * e], s[c + 2 * e + 1]);
      const float mx = fmaxf(max3(x[0], x[1], x[2]), x[3]) * sl2;
      const bool grow = mx > m + kGrow || (m == -CUDART_INF_F && mx > m);
      if (__any_sync(0xffffffffu, grow)) {
        const float f = grow ? ex2(m - mx) : 1.f;   // m = -inf: 0
        if (grow) m = mx;
        sum[0] = mul2(sum[0], pair(f, f)), sum[1] = mul2(sum[1], pair(f, f));
        if (i > 0) {   // O as of tile i - 1
          if (!__all_sync(0xffffffffu, bar_wait<0>(&sh.pv_done[b ^ 1], ((i - 1) >> 1) & 1, fail, &g_prefill_attn_status, WAIT_PV))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
          for (int c = 0; c < D; c += 8) {
            uint32_t o[8];
            tmem_ld8(tq + kO + c, o);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
            tmem_st8(tq + kO + c, o);
          }
        }
      }
      const float sub = m == -CUDART_INF_F ? 0.f : -m;   // nothing visible yet: every probability is 2^-inf
      const uint64_t sub2 = pair(sub, sub), scale2 = pair(sl2, sl2);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t p[kTile / 4], r[kTile / 4];   // fp16 values and remainders
#pragma unroll
        for (int c = 0; c < kTile / 2; c += 2) {
          float u, v;
          unpair(fma2(pair(s[kTile / 2 * h + c], s[kTile / 2 * h + c + 1]), scale2, sub2), u, v);
          u = ex2(u), v = ex2(v);
          sum[(c >> 1) & 1] = add2(sum[(c >> 1) & 1], pair(u, v));
          const half2 hi = __floats2half2_rn(u, v);
          const float2 f = __half22float2(hi);
          p[c / 2] = as_u32(hi);
          r[c / 2] = as_u32(__floats2half2_rn(u - f.x, v - f.y));
        }
        tmem_st16(ts + (uint32_t)(kTile / 4 * h), p);   // over the scores: values, then remainders
        tmem_st16(ts + (uint32_t)(kTile / 2 + kTile / 4 * h), r);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&sh.p_full[b]);
    }
    float l0, l1, l2, l3;
    unpair(sum[0], l0, l1), unpair(sum[1], l2, l3);
    l = (l0 + l1) + (l2 + l3);
  } else if (warp == kMmaWarp) {
    // M = 128; S: N = 64, both operands K-major; O: N = D, B (V) MN-major (bit 16)
    constexpr uint32_t idesc_s = (1u << 4) | ((kTile >> 3) << 17) | ((128u >> 4) << 24);
    constexpr uint32_t idesc_o = (1u << 4) | (1u << 16) | ((D >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t q_s = sa(base), ring_s = sa(ring);
    auto scores = [&](int i) {   // S of tile i
      const uint32_t k_s = ring_s + (i % NS) * TILE;
#pragma unroll
      for (int k = 0; k < D / 16; ++k)
        mma_ss(tmem + (uint32_t)(kTile * (i & 1)), desc_sw128(q_s + (k / 4) * (kRows * 128)) + 2 * (k % 4),
               desc_sw128(k_s + (k / 4) * (kTile * 128)) + 2 * (k % 4), idesc_s, k > 0);
      commit(&sh.s_full[i & 1]);
      commit(&sh.k_empty[i % NS]);
    };
    auto arrived = [&](uint64_t* bar, uint32_t parity, int code) {
      const bool ok = __all_sync(0xffffffffu, bar_wait<0>(bar, parity, fail, &g_prefill_attn_status, code));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    bool ok = ntiles > 0 && arrived(&sh.q_full, 0, WAIT_Q);
    for (int i = 0; i < min(2, ntiles) && ok; ++i)
      if ((ok = arrived(&sh.k_full[i], 0, WAIT_K))) scores(i);
#pragma unroll 1
    for (int i = 0; i < ntiles && ok; ++i) {
      const int n = i + 2;
      ok = arrived(&sh.v_full[i % NS], (i / NS) & 1, WAIT_V) && (n >= ntiles || arrived(&sh.k_full[n % NS], (n / NS) & 1, WAIT_K)) &&
           arrived(&sh.p_full[i & 1], (i >> 1) & 1, WAIT_P);
      if (!ok) break;
      const uint32_t v_s = ring_s + (NS + i % NS) * TILE;
#pragma unroll
      for (int k = 0; k < kTile / 8; ++k)   // values, then remainders, both against all of V
        mma_ts(tmem + kO, tmem + (uint32_t)(kTile * (i & 1) + 8 * k), desc_sw128(v_s, kTile * 128) + 128 * (k % (kTile / 16)), idesc_o,
               i > 0 || k > 0);
      commit(&sh.pv_done[i & 1]);
      if (n < ntiles) scores(n);   // over the scores and probabilities of tile i, behind the product that reads them
      commit(&sh.v_empty[i % NS]);
    }
    commit(&sh.drain);   // whatever was issued has completed before the CTA's memory goes away
    bool done = false;
    for (int i = 0; i < (1 << 16) && !(done = bar_try(&sh.drain, 0)); ++i) __nanosleep(32);
    if (!done) *fail = 1, atomicCAS(&g_prefill_attn_status, 0, WAIT_DRAIN);
  } else {
    // Half the warps copy K, half V; a warp takes RW rows of a tile, 32 / PP at a time, and hands a tile over when it has issued
    // kLag more. (One TMA box per page instead: 80 ns a box of 2 KB, a third slower in all.)
    constexpr int IT = 16;
    static_assert(RW * PP == 32 * IT, "16 copies a lane and tile");
    const int w = warp - kMmaWarp - 1, p = lane % PP;   // K: even warps
    const bool is_v = w & 1;
    uint64_t *full = is_v ? sh.v_full : sh.k_full, *empty = is_v ? sh.v_empty : sh.k_empty;
    const half* from = (is_v ? vc : kc) + 8 * p;
    const uint32_t at = sa(ring) + (is_v ? NS * TILE : 0) + first * 128;
    uint32_t to[8 / (32 / PP)];   // rows 8 apart have one position in the swizzle
#pragma unroll
    for (int k = 0; k < 8 / (32 / PP); ++k) to[k] = at + swz_piece(lane / PP + k * (32 / PP), p, kTile);
    auto hand_over = [&](int i) {   // this warp's part of tile i has landed
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(&full[i % NS]);
    };
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < ntiles; ++i) {
      const int a = lo, b = hi, n = min(i + 1, ntiles - 1);
      lo = row(n, lane), hi = RW > 32 ? row(n, lane + 32) : 0;
      ok = i < NS || __all_sync(0xffffffffu, bar_wait<32>(&empty[i % NS], (i / NS - 1) & 1, fail, &g_prefill_attn_status, WAIT_STAGE));
      if (!ok) break;
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        const int r = k * (32 / PP);
        const int off = __shfl_sync(0xffffffffu, r < 32 ? a : b, (r & 31) + lane / PP);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to[k % (8 / (32 / PP))] + (i % NS) * TILE + (r & ~7) * 128),
                     "l"(from + (size_t)off * D)
                     : "memory");
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
  float* park = reinterpret_cast<float*>(base);               // [kRows][OP], over Q and the idle stages
  float2* ml = reinterpret_cast<float2*>(park + kRows * OP);  // [kRows]
  static_assert(kRows * OP * 4 + kRows * 8 <= kRows * D * 2 + 2 * NS * TILE, "partials fit over the stages");
  if (warp < kSoftWarps && !*fail) {
    const int r = row0 + tid, t = r >> log2hpg, h = (kvh << log2hpg) + (r & (hpg - 1));
    const float f = C == 1 ? 1.f / l : 1.f;
    half2 any = __float2half2_rn(0.f);   // NaN if one of the row is (or if infinities of both signs are: redo_row looks closer)
    half* o = out + ((size_t)t * n_q + h) * D;
#pragma unroll 1
    for (int c = 0; c < D; c += 16) {
      uint32_t v[16];
      if (ntiles > 0) {
        tmem_ld16(tq + kO + c, v);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) v[e] = 0u;
      }
      if (C == 1) {
        uint32_t u[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) u[e] = as_u32(__floats2half2_rn(__uint_as_float(v[2 * e]) * f, __uint_as_float(v[2 * e + 1]) * f));
        if (t < T) {
          reinterpret_cast<uint4*>(o + c)[0] = make_uint4(u[0], u[1], u[2], u[3]);
          reinterpret_cast<uint4*>(o + c)[1] = make_uint4(u[4], u[5], u[6], u[7]);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) any = __hadd2(any, as_h2(u[e]));
      } else {
#pragma unroll
        for (int e = 0; e < 16; e += 4)
          *reinterpret_cast<uint4*>(park + tid * OP + c + e) = make_uint4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      }
    }
    ml[tid] = make_float2(m, l);
    if (t < T && (__hisnan(__low2half(any)) || __hisnan(__high2half(any))))
      redo_row<D>(RowArgs{q + (size_t)t * q_stride + (size_t)h * D, kc, vc, bt, kvh, n_kv, log2P, start + t, last, sl2, o}, 0, D);
  }
  if (C > 1) {
    cluster_barrier();
    if (!*fail) {   // CTA `split` finishes every C-th row; a thread takes four dims
      for (int i = tid; i < kRows / C * (D / 4); i += threads<D>()) {
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
        if (t < T) {
          const int h = (kvh << log2hpg) + (r & (hpg - 1));
          half* to = out + ((size_t)t * n_q + h) * D + d;
          *reinterpret_cast<uint2*>(to) = make_uint2(as_u32(__floats2half2_rn(o.x * f, o.y * f)), as_u32(__floats2half2_rn(o.z * f, o.w * f)));
          const float any = (o.x + o.y + o.z + o.w) * f;
          if (any != any)
            redo_row<D>(RowArgs{q + (size_t)t * q_stride + (size_t)h * D, kc, vc, bt, kvh, n_kv, log2P, start + t, last, sl2, to - d}, d, d + 4);
        }
      }
    }
    cluster_barrier();   // nobody's shared memory goes away while a peer still reads it
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemColumns) : "memory");
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
  // one wave of CTAs, four tiles each at least so that a split outweighs its merge (~2 us; at two, 200 tokens: 6.3 -> 8.1 us)
  const int slots = 2 * kNumSMs;
  int C = 1;
  while (C < kMaxSplit && row_blocks * n_kv * C * 2 <= slots && tiles >= 4 * 2 * C) C *= 2;
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
  cfg.gridDim = dim3(row_blocks * n_kv, 1, C);
  cfg.blockDim = dim3(D == 64 ? threads<64>() : threads<128>());
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, (const half*)q, q_stride, (const half*)kc, (const half*)vc, bt, start, T, n_kv, log2hpg, log2P,
                            1.44269504088896340736f / sqrtf((float)D), (half*)out);
}

}  // namespace b200
