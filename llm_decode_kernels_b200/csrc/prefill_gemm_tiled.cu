// Prompt GEMM from the tile layout:  Y[T, N] = X[T, K] . dequant(W)[N, K]^T for any number of tokens, optionally with SwiGLU
// (paired [gate; up] layout), fp32 accumulation, fp16 out. The fp16 weights are the format's (dequant_w4a16_kernel), bit for bit.
//
// What bounds a W4A16 GEMM here is not the tensor core but what has to reach it: with a 128-row tile per CTA every 64 columns of
// K bring 32 KB of activations (256 tokens) from the L2 for 512 cycles of MMA, more than the L2 delivers to 148 SMs, and the
// dequantized weights (16 KB) pass through shared memory twice. So:
//   * two CTAs on neighbouring SMs work as a pair (cta_group::2): 256 rows of W x up to 256 tokens, each CTA brings 128 rows of
//     W and half of the tokens - half the activation traffic per MMA cycle;
//   * the dequantized weights never touch shared memory: a dequantizing thread owns a row, its tcgen05.st puts the row's fp16 pairs
//     into tensor memory, and the MMA reads its A operand there;
//   * a CTA pair is persistent: it walks over output tiles, the dequantizing and copying warps run four to six 128-column units
//     ahead across tile borders, and the epilogue warps empty the accumulator into shared memory (rounded to fp16) before they
//     store, so the next tile's MMAs wait only for that; the CTA's last tile is emptied and stored by all warps;
//   * where there are fewer tiles than pairs, S = 2 or 4 pairs (one cluster) share a tile by splitting K; their fp32 partial tiles
//     are written into the shared memory of the CTA that finishes a token and added there in a fixed order.
// What follows the product in a prompt rides in the epilogue (MODE): SwiGLU, the residual row with the next norm's input and sums, RoPE
// and the append to the cache; and the norm's factor, which is applied to fp32 outputs.
// Warps: 0-11 dequantize (three groups of four, every third unit: a unit is ~2000 cycles of latency for a warp and 1024 of MMA at
// 256 tokens), 12-15 epilogue, 16 MMA issue (even CTA of a pair), 17 TMA.
// Tensor memory: accumulator (128 lanes = rows, one column per token; 128 or 256 columns), then six or four A stages of 64 columns.
// Loops that run once per launch at small sizes are kept short rather than unrolled: every launch fetches its code anew.
// Every wait is bounded; a wait that runs out raises the CTA's fail flag, all roles leave, the CTA waits (bounded) for its copies,
// joins the cluster barriers, frees its tensor memory, and b200_gemm_w4a16_status is non-zero.
#include "common.cuh"
#include "prefill.h"
#include "umma.cuh"

namespace b200 {

namespace {

using namespace umma;

__device__ int g_tiled_status = 0;   // 0, or the code of the first wait inside prefill_gemm_tiled_kernel that ran out

constexpr int kDqGroups = 3, kDqWarps = 4 * kDqGroups, kEpWarps = 4, kThreads = (kDqWarps + kEpWarps + 2) * 32;
constexpr int kMmaWarp = kDqWarps + kEpWarps, kTmaWarp = kMmaWarp + 1;
constexpr int kMaxStages = 6;          // 128-column units in flight: A in tensor memory, B in shared memory
constexpr int kACols = 64;             // tensor-memory columns of an A stage
constexpr int kMaxTokens = 256;        // tokens per tile = N of the MMA (a multiple of 32)
constexpr int kMaxSplit = 4;           // pairs per tile: clusters of at most 8 CTAs
// Units of K that one accumulator sums: the tensor core drops bits at every step of a chain. Error against 64 bits at K = 28672 (224
// units): 2.097e-4 in one chain, 2.077e-4 in two, of which 2.070e-4 is the rounding of the output; up to K = 8192 one chain loses
// nothing (2.0758e-4 and 2.0736e-4). Longer rows are split whatever the cost rule says.
constexpr int kMaxChain = 112;
enum : int { WAIT_DQ = 1, WAIT_MMA_ACC = 2, WAIT_MMA_FULL = 3, WAIT_TMA = 5, WAIT_EP = 6 };

// one arrival on `bar` in both CTAs of the pair when the MMAs issued so far by the elected lane have completed (whole warp)
DEVI void commit_pair(uint64_t* bar, uint32_t ctas) {
  asm volatile(
      "{\n\t.reg .pred e;\n\t.reg .b16 m;\n\t"
      "cvt.u16.u32 m, %1;\n\t"
      "elect.sync _|e, 0xffffffff;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(sa(bar)),
      "r"(ctas)
      : "memory");
}

template <int SLEEP_NS>
DEVI bool bar_wait(uint64_t* b, uint32_t parity, volatile int* fail, int code) {
  return umma::bar_wait<SLEEP_NS>(b, parity, fail, &g_tiled_status, code);
}

struct Shared {
  uint64_t full[kMaxStages], empty[kMaxStages], acc_full, acc_empty;
  uint32_t tmem;
  int fail;
  float top[kEpWarps];   // norm_top
};

// Stage and how often it has been used before, of a sequence that takes the stages in turn.
struct Ring {
  int s, use;
  DEVI void step(int n, int stages) {
    s += n;
    if (s >= stages) s -= stages, ++use;
  }
};

// one row's 128 weights of a unit and their (scale, zero)
struct RowUnit { uint4 w[4]; half2 sz; };

DEVI void ld32(const uint8_t* p, uint4& a, uint4& b) {   // one whole 32-byte sector per lane
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
               : "l"(p));
}

// (q - z) * s per pair of weights, as dequant_w4a16_kernel. Nibbles at bits 0-3 / 16-19 become 1024 + q, those at bits 4-7 / 20-23
// where they stand 64 + q (ulp 1 and 1/16: both exact), and 64 + z is made of what 1024 + z rounds z to: the same difference, bit for
// bit, without a shift. (As 1024 + 16 q and s / 16, which a subnormal s does not survive, it took a second form of the loop and a vote
// between the two: 0.35 instead of 0.30 us a unit.)
DEVI half2 nib_hi64(uint32_t w) { return as_h2((w & 0x00F000F0u) | 0x54005400u); }
DEVI void dequant_store(const RowUnit& d, uint32_t dst) {
  const half2 z2 = __half2half2(__high2half(d.sz)), s2 = __half2half2(__low2half(d.sz));
  const half2 k1024 = __float2half2_rn(1024.f), zl = __hadd2(z2, k1024), zh = __hadd2(__hsub2(zl, k1024), __float2half2_rn(64.f));
#pragma unroll
  for (int h = 0; h < 4; ++h) {   // 32 columns of K = 16 columns of tensor memory
    const uint32_t w4[4] = {d.w[h].x, d.w[h].y, d.w[h].z, d.w[h].w};
    uint32_t o[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t w = w4[j], wh = w >> 8;
      o[4 * j] = as_u32(__hmul2(__hsub2(nib_lo(w), zl), s2));
      o[4 * j + 1] = as_u32(__hmul2(__hsub2(nib_hi64(w), zh), s2));
      o[4 * j + 2] = as_u32(__hmul2(__hsub2(nib_lo(wh), zl), s2));
      o[4 * j + 3] = as_u32(__hmul2(__hsub2(nib_hi64(wh), zh), s2));
    }
    tmem_st16(dst + 16 * h, o);
  }
}

// half(silu(gate)) * up for two outputs, the rounding points of swiglu_kernel
DEVI uint32_t gated2(uint32_t gate, uint32_t up) {
  const float2 g = __half22float2(as_h2(gate));
  const half2 s = __floats2half2_rn(__fdividef(g.x, 1.f + __expf(-g.x)), __fdividef(g.y, 1.f + __expf(-g.y)));
  return as_u32(__hmul2(s, as_h2(up)));
}

// what the epilogue multiplies a token's outputs by: the norm's factor rsqrt(mean square + eps), and what its row of X lacks beside it
DEVI float token_factor(const PrefillNorm& nm, int t) {
  float a = 0.f, b = 0.f;   // two chains, always the same order
  const float* p = nm.ss_in + (size_t)t * nm.parts;
#pragma unroll 8
  for (int i = 0; i + 1 < nm.parts; i += 2) a += p[i], b += p[i + 1];
  if (nm.parts & 1) a += p[nm.parts - 1];
  return rsqrtf((a + b) * nm.inv_h + nm.eps) * nm.inv_in[t];
}

// The largest |w| of the next norm, each warp's of the epilogue (thread et of their 128) in sh.top; norm_scale: the p made of it (PrefillNorm). w is
// none of the chunk's outputs: read ahead of the wait, while the first units are on their way. (NaN is no maximum; its column is NaN anyway.)
DEVI void norm_top(const PrefillNorm& nm, int N, Shared& sh, int et) {
  float m = 0.f;
#pragma unroll 4
  for (int i = et; i < N >> 3; i += 32 * kEpWarps) {
    float f[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(nm.w) + i), f);
#pragma unroll
    for (int k = 0; k < 8; ++k) m = fmaxf(m, fabsf(f[k]));
  }
  m = warp_max(m);
  if ((et & 31) == 0) sh.top[et >> 5] = m;
}
DEVI float norm_scale(const Shared& sh) { return pow2_above(fmaxf(fmaxf(sh.top[0], sh.top[1]), fmaxf(sh.top[2], sh.top[3]))); }

// Eight columns of a finished residual row: x += y, xw = x * w * scale; returns the sum of x^2.
DEVI float residual8(const uint4& r, const uint4& y, const uint4& w, half* x, half* xw, float scale) {   // r: x as it was
  const uint32_t yu[4] = {y.x, y.y, y.z, y.w}, wu[4] = {w.x, w.y, w.z, w.w};
  uint32_t ru[4] = {r.x, r.y, r.z, r.w}, o[4];
  float ss = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    ru[e] = as_u32(__hadd2(as_h2(ru[e]), as_h2(yu[e])));
    const float2 f = __half22float2(as_h2(ru[e])), g = __half22float2(as_h2(wu[e]));
    ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
    o[e] = as_u32(__floats2half2_rn(f.x * g.x * scale, f.y * g.y * scale));
  }
  *reinterpret_cast<uint4*>(x) = make_uint4(ru[0], ru[1], ru[2], ru[3]);
  *reinterpret_cast<uint4*>(xw) = make_uint4(o[0], o[1], o[2], o[3]);
  return ss;
}

// The accumulator of a CTA's 128 rows x nt tokens -> rows[token pair][128 rows], two tokens of a row in a word: columns c0 .. c0 + 31 of
// every `step`, by a warp that reaches lanes 32 q .. . The next tile's MMAs wait for this: with a token's row as a half of its own
// (single conversions, 2-byte stores) it took 1.8 us for 128 tokens, a quarter of a tile's time at 256.
DEVI void park_tile(uint32_t tmem, int q, int lane, uint32_t* rows, int c0, int step, int nt, const float* fac) {
  const uint32_t from = tmem + ((uint32_t)(32 * q) << 16);
#pragma unroll 1
  for (int c = c0; c < nt; c += step) {   // nt is a multiple of 32
    float v[32];
    tmem_ld16_async(from + c, v);
    tmem_ld16_async(from + c + 16, v + 16);
    tmem_wait_ld(v);
    if (fac) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 f = *reinterpret_cast<const float4*>(fac + c + j);
        v[j] *= f.x, v[j + 1] *= f.y, v[j + 2] *= f.z, v[j + 3] *= f.w;
      }
    }
    uint32_t* to = rows + (c >> 1) * 128 + 32 * q + lane;
#pragma unroll
    for (int j = 0; j < 16; ++j) to[128 * j] = as_u32(__floats2half2_rn(v[2 * j], v[2 * j + 1]));
  }
}

// rows -> Y: tokens t0 .. of the tile, features from row0 (SWIGLU: half of it) on; thread `at` of `threads`. A thread takes eight outputs of
// two tokens.
template <bool SWIGLU>
DEVI void store_tile(const uint32_t* rows, half* Y, int T, int N, int t0, int row0, int nt, int at, int threads) {
  constexpr int kPieces = SWIGLU ? 8 : 16;   // pieces of 8 outputs per token
  const bool vec = (N & 7) == 0 && (reinterpret_cast<uintptr_t>(Y) & 15) == 0;
  const int pairs = (min(nt, T - t0) + 1) >> 1;
#pragma unroll 1
  for (int i = at; i < pairs * kPieces; i += threads) {
    const int tp = i / kPieces, pc = i % kPieces, f = (SWIGLU ? row0 >> 1 : row0) + 8 * pc;
    const uint4* src = reinterpret_cast<const uint4*>(rows + tp * 128 + (SWIGLU ? 16 : 8) * pc);
    const uint4 a = src[0], b = src[1];
    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    if (SWIGLU) {   // rows 16 k + 0..7 are gates, 16 k + 8..15 their up rows
      const uint4 c = src[2], d = src[3];
      const uint32_t u[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = gated2(w[e], u[e]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = t0 + 2 * tp + h;
      if (t >= T) break;
      uint32_t o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = __byte_perm(w[2 * e], w[2 * e + 1], h ? 0x7632 : 0x5410);
      half* y = Y + (size_t)t * N + f;
      if (vec && f + 7 < N) {
        *reinterpret_cast<uint4*>(y) = make_uint4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (f + e < N) y[e] = __ushort_as_half((unsigned short)(o[e >> 1] >> (16 * (e & 1))));
      }
    }
  }
}

// rows -> the residual stream (PrefillNorm): 16 lanes take a token pair's 128 columns, so each of the two sums is one of theirs.
DEVI void store_residual(const uint32_t* rows, const PrefillNorm& nm, float p, int T, int N, int t0, int row0, int nt, int at, int threads) {
  const int lane = at & 31, pairs = (min(nt, T - t0) + 1) >> 1, pc = at & 15, f = row0 + 8 * pc;
  if (row0 >= N) return;   // N is a multiple of 128
  const uint4 w8 = __ldg(reinterpret_cast<const uint4*>(nm.w + f));
  const float scale = 1.f / p;
  uint4 next[2];   // the pair's rows of x, one round ahead
  auto fetch = [&](int i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = t0 + 2 * (i >> 4) + h;
      if ((i >> 4) < pairs && t < T) next[h] = *reinterpret_cast<const uint4*>(nm.x + (size_t)t * N + f);
    }
  };
  fetch(at);
#pragma unroll 1
  for (int i = at; i - lane < pairs * 16; i += threads) {
    const int tp = i >> 4;
    float ss[2] = {0.f, 0.f};
    const uint4 was[2] = {next[0], next[1]};
    fetch(i + threads);
    if (tp < pairs) {
      const uint4* src = reinterpret_cast<const uint4*>(rows + tp * 128 + 8 * pc);
      const uint4 a = src[0], b = src[1];
      const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = t0 + 2 * tp + h;
        if (t < T) {
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) o[e] = __byte_perm(w[2 * e], w[2 * e + 1], h ? 0x7632 : 0x5410);
          ss[h] = residual8(was[h], make_uint4(o[0], o[1], o[2], o[3]), w8, nm.x + (size_t)t * N + f, nm.xw + (size_t)t * N + f, scale);
        }
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], o);
      ss[1] += __shfl_xor_sync(0xffffffffu, ss[1], o);
    }
    const int t = t0 + 2 * tp + pc;   // lanes 0 and 1 of the sixteen
    if (tp < pairs && pc < 2 && t < T) {
      nm.ss_out[(size_t)t * nm.parts + (row0 >> 7)] = pc ? ss[1] : ss[0];
      if (row0 == 0) nm.inv_out[t] = p;
    }
  }
}

// Where head `head` of token t goes from its first dim on: rotated q to Y, k and v to their row of the cache.
DEVI half* head_row(const PrefillRope& rp, half* Y, int N, int head, int t, int page, int slot) {
  if (head < rp.n_q) return Y + (size_t)t * N + head * rp.D;
  const bool k = head < rp.n_q + rp.n_kv;
  const int kvh = head - rp.n_q - (k ? 0 : rp.n_kv);
  return (k ? rp.kc : rp.vc) + ((((size_t)page * rp.n_kv + kvh) << rp.log2P) + slot) * rp.D;
}

// rows -> q, K and V: a thread takes eight rotation pairs of two tokens (128 rows are whole heads: two of 64 dims or one of 128).
DEVI void store_rope(const uint32_t* rows, const PrefillRope& rp, const int* positions, half* Y, int T, int N, int t0, int row0, int nt, int at, int threads) {
  const int pairs = (min(nt, T - t0) + 1) >> 1, d2 = rp.D >> 1, heads = rp.n_q + 2 * rp.n_kv;
#pragma unroll 1
  for (int i = at; i < pairs * 8; i += threads) {
    const int tp = i >> 3, j = 8 * (i & 7), local = j & (d2 - 1), lo_row = (j & ~(d2 - 1)) * 2 + local;   // pair j of the 64 of these rows
    const int head = (row0 + lo_row) / rp.D;
    if (head >= heads) continue;
    const bool rotate = head < rp.n_q + rp.n_kv;
    const int pos[2] = {positions[2 * tp], positions[2 * tp + 1]};   // of a token behind the last: the last one's
    float4 cs[2][2], sn[2][2];   // both tokens' factors are in flight together
    int page[2] = {0, 0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (rotate) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          cs[h][v] = __ldg(reinterpret_cast<const float4*>(rp.cos_t + (size_t)pos[h] * d2 + local) + v);
          sn[h][v] = __ldg(reinterpret_cast<const float4*>(rp.sin_t + (size_t)pos[h] * d2 + local) + v);
        }
      }
      if (head >= rp.n_q) page[h] = __ldg(rp.bt + (pos[h] >> rp.log2P));
    }
    const uint4 *lp = reinterpret_cast<const uint4*>(rows + tp * 128 + lo_row), *hp = reinterpret_cast<const uint4*>(rows + tp * 128 + lo_row + d2);
    const uint4 l0 = lp[0], l1 = lp[1], h0 = hp[0], h1 = hp[1];
    const uint32_t lw[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w}, hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int t = t0 + 2 * tp + h;
      uint32_t lo[4], hi[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t sel = h ? 0x7632 : 0x5410;
        lo[e] = __byte_perm(lw[2 * e], lw[2 * e + 1], sel), hi[e] = __byte_perm(hw[2 * e], hw[2 * e + 1], sel);
      }
      if (rotate) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const float4 c = cs[h][v], s = sn[h][v];
          const float2 a01 = __half22float2(as_h2(lo[2 * v])), a23 = __half22float2(as_h2(lo[2 * v + 1]));
          const float2 b01 = __half22float2(as_h2(hi[2 * v])), b23 = __half22float2(as_h2(hi[2 * v + 1]));
          lo[2 * v] = as_u32(__floats2half2_rn(a01.x * c.x - b01.x * s.x, a01.y * c.y - b01.y * s.y));
          lo[2 * v + 1] = as_u32(__floats2half2_rn(a23.x * c.z - b23.x * s.z, a23.y * c.w - b23.y * s.w));
          hi[2 * v] = as_u32(__floats2half2_rn(b01.x * c.x + a01.x * s.x, b01.y * c.y + a01.y * s.y));
          hi[2 * v + 1] = as_u32(__floats2half2_rn(b23.x * c.z + a23.x * s.z, b23.y * c.w + a23.y * s.w));
        }
      }
      if (t >= T) break;
      half* to = head_row(rp, Y, N, head, t, page[h], pos[h] & ((1 << rp.log2P) - 1)) + local;
      *reinterpret_cast<uint4*>(to) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
      *reinterpret_cast<uint4*>(to + d2) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    }
  }
}

enum : int { PLAIN, GATED, RESIDUAL, ROPE };   // what the epilogue does: Y as it is, SwiGLU, PrefillNorm's residual row, PrefillRope

}  // namespace

template <int MODE>
__global__ void __launch_bounds__(kThreads, 1)
prefill_gemm_tiled_kernel(const __grid_constant__ CUtensorMap xmap, const uint8_t* __restrict__ Wt, half* __restrict__ Y, int T,
                          int N, int row_tiles, int nunit, int nt, int S, int feat_tiles, int tiles, int ns, int p_apart, const PrefillNorm nm, const PrefillRope rp) {
  extern __shared__ uint8_t raw[];
  __shared__ Shared sh;
  __shared__ __align__(16) float token_fac[MODE == RESIDUAL ? 4 : kMaxTokens];
  __shared__ int token_pos[MODE == ROPE ? kMaxTokens : 1];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // warp: known to be uniform
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int csize = 2 * S, first = blockIdx.x / csize, stride = gridDim.x / csize;
  const int split = rank >> 1, side = rank & 1;            // which share of K; which half of the pair
  const uint32_t lead = rank & ~1u;
  const int u0 = nunit * split / S, u1 = nunit * (split + 1) / S;
  const int half_bytes = nt * 64, stage_bytes = 2 * half_bytes;   // 64 columns of K x nt / 2 tokens; a unit
  uint32_t* rows = reinterpret_cast<uint32_t*>(base + ns * stage_bytes);   // a finished tile, see park_tile
  const float* fac = MODE != RESIDUAL && nm.ss_in ? token_fac : nullptr;   // multiplies the outputs
  volatile int* fail = &sh.fail;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(sa(&sh.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&xmap) : "memory");   // before the wait for X, not behind it
    for (int s = 0; s < ns; ++s) {
      bar_init(&sh.full[s], 2 * 4 + 1);   // one group of dequantizing warps in each CTA of the pair, and the copies
      bar_init(&sh.empty[s], 1);
    }
    bar_init(&sh.acc_full, 1);
    bar_init(&sh.acc_empty, 2 * kEpWarps);
    sh.fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_barrier();   // the peers' barriers exist before anything arrives on them
  // only now, with its tensor memory allocated: a dependent CTA that got there first and then waited for this grid would not give
  // it back
  pdl_launch_dependents();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem, tmem_a = tmem + (uint32_t)(512 - kACols * ns);

  if (warp < kDqWarps) {
    // ---- A: thread = row; group `grp` takes every third unit of the sequence, with the next two in registers
    const int grp = warp >> 2, r = (warp & 3) * 32 + lane;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const int nu = u1 - u0, total = first < tiles ? ((tiles - 1 - first) / stride + 1) * nu : 0;   // units of this CTA's sequence
    // the unit loaded next: its place in the sequence and in its tile, and where this row's weights of it are (null past the matrix)
    int li = grp, lu = grp, ltile = first;
    const uint8_t* lp;
    auto seek = [&] {
      const int rt = 16 * (ltile % feat_tiles) + 8 * side + (r >> 4);
      lp = ltile < tiles && rt < row_tiles ? Wt + ((size_t)rt * nunit + u0 + lu) * kTileUnitBytes : nullptr;
    };
    auto wrap = [&] {
      while (lu >= nu) lu -= nu, ltile += stride;
      seek();
    };
    wrap();
    auto load = [&](RowUnit& d) {
      if (lp && li < total) {
        const uint8_t* q = lp + 64 * (r & 15);
        ld32(q, d.w[0], d.w[1]);
        ld32(q + 32, d.w[2], d.w[3]);
        d.sz = __ldg(reinterpret_cast<const half2*>(lp + 1024) + (r & 15));
      } else {   // rows past the matrix: zero words, zero scale
#pragma unroll
        for (int i = 0; i < 4; ++i) d.w[i] = make_uint4(0u, 0u, 0u, 0u);
        d.sz = __float2half2_rn(0.f);
      }
      li += kDqGroups;
      lu += kDqGroups;
      if (lu >= nu) wrap();
      else if (lp) lp += kDqGroups * kTileUnitBytes;
    };
    RowUnit cur, next, after;
    load(cur);
    load(next);
    Ring ring = {grp, 0};
    const uint32_t full0 = in_cta(sa(&sh.full[0]), lead);
#pragma unroll 1
    for (int i = grp; i < total; i += kDqGroups) {
      load(after);
      if (ring.use > 0 && !__all_sync(0xffffffffu, bar_wait<64>(&sh.empty[ring.s], (ring.use - 1) & 1, fail, WAIT_DQ))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t dst = tmem_a + lanes + (uint32_t)(kACols * ring.s);
      dequant_store(cur, dst);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive_cluster(full0 + 8 * ring.s);
      ring.step(kDqGroups, ns);
      cur = next;
      next = after;
    }
  } else if (warp == kMmaWarp) {
    if (side == 0) {
      // The whole warp runs the loop and one elected lane issues. In code that only one lane enters the compiler cannot keep the
      // descriptors in uniform registers, and the eight MMAs of a unit took 580 cycles to issue, more than they take to run.
      // D fp32, A and B fp16, both K-major, N / 8 in bits 17-22, M / 16 in bits 24-28 (M = 256 over the pair)
      const uint32_t idesc = (1u << 4) | ((uint32_t)(nt >> 3) << 17) | ((256u >> 4) << 24);
      const uint32_t both = 3u << lead;
      bool ok = true;
      int done = 0;
      Ring ring = {0, 0};
#pragma unroll 1
      for (int tile = first; tile < tiles && ok; tile += stride, ++done) {
        if (done > 0) ok = __all_sync(0xffffffffu, bar_wait<0>(&sh.acc_empty, (done - 1) & 1, fail, WAIT_MMA_ACC));
#pragma unroll 1
        for (int u = u0; u < u1 && ok; ++u) {
          ok = __all_sync(0xffffffffu, bar_wait<0>(&sh.full[ring.s], ring.use & 1, fail, WAIT_MMA_FULL));
          if (!ok) break;
          const uint32_t a = tmem_a + (uint32_t)(kACols * ring.s), bs = sa(base + ring.s * stage_bytes);
          asm volatile(
              "{\n\t.reg .pred e, p;\n\t.reg .b32 a1;\n\t.reg .b64 d;\n\t"
              "tcgen05.fence::after_thread_sync;\n\t"
              "elect.sync _|e, 0xffffffff;\n\t"
              "setp.ne.b32 p, %5, 0;\n\t"
              "@e tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %4, p;\n\t"
              "setp.eq.b32 p, 0, 0;\n\t"
              "add.u32 a1, %1, 8;\n\tadd.u64 d, %2, 2;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d, %4, p;\n\t"
              "add.u32 a1, %1, 16;\n\tadd.u64 d, %2, 4;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d, %4, p;\n\t"
              "add.u32 a1, %1, 24;\n\tadd.u64 d, %2, 6;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d, %4, p;\n\t"
              "add.u32 a1, %1, 32;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], %3, %4, p;\n\t"
              "add.u32 a1, %1, 40;\n\tadd.u64 d, %3, 2;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d, %4, p;\n\t"
              "add.u32 a1, %1, 48;\n\tadd.u64 d, %3, 4;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d, %4, p;\n\t"
              "add.u32 a1, %1, 56;\n\tadd.u64 d, %3, 6;\n\t@e tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], d, %4, p;\n\t"
              "}" ::"r"(tmem),
              "r"(a), "l"(desc_sw128(bs)), "l"(desc_sw128(bs + half_bytes)), "r"(idesc), "r"(u > u0 ? 1u : 0u)
              : "memory");
          commit_pair(&sh.empty[ring.s], both);
          ring.step(1, ns);
        }
        if (ok) commit_pair(&sh.acc_full, both);
      }
    }
  } else if (warp == kTmaWarp) {
    pdl_wait();   // X is the predecessor's output
    {
      // What a unit costs this warp is what few tokens pay a unit, as for the MMA warp: one barrier for both operands, the token offset
      // (a division) once a tile. Like the MMA warp, all lanes run the loop; one copy brings both 64-column halves of a unit (a third dimension of the tensor
      // map). Two copies a unit from a single-lane branch took 440 cycles of the pair's 970 per unit at few tokens.
      Ring ring = {0, 0};
      bool ok = true;
      const uint32_t full0 = in_cta(sa(&sh.full[0]), lead), own0 = sa(&sh.full[0]), dst0 = sa(base);   // both CTAs' halves count on the even CTA's barrier
#pragma unroll 1
      for (int tile = first; tile < tiles && ok; tile += stride) {
        const int y = (tile / feat_tiles) * nt + side * (nt >> 1);
#pragma unroll 1
        for (int u = u0; u < u1; ++u) {
          if (ring.use > 0 && !__all_sync(0xffffffffu, bar_wait<0>(&sh.empty[ring.s], (ring.use - 1) & 1, fail, WAIT_TMA))) {
            ok = false;
            break;
          }
          asm volatile(
              "{\n\t.reg .pred e, l;\n\t"
              "elect.sync _|e, 0xffffffff;\n\t"
              "setp.eq.and.b32 l, %6, 0, e;\n\t"
              "@l mbarrier.arrive.expect_tx.shared::cta.b64 _, [%7], %8;\n\t"
              "@e cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
              "[%5];\n\t}" ::"r"(dst0 + ring.s * stage_bytes),
              "l"(&xmap), "r"(0), "r"(y), "r"(2 * u), "r"(full0 + 8 * ring.s), "r"(side), "r"(own0 + 8 * ring.s), "r"((uint32_t)(2 * stage_bytes))
              : "memory");
          ring.step(1, ns);
        }
      }
      // giving up: let the copies in flight land before the shared memory goes away (the even CTA holds the barriers)
      if (*fail && side == 0 && lane == 0)
        for (int s = 0; s < ns; ++s) {
          const int uses = ring.use + (s < ring.s ? 1 : 0);   // how often stage s has been filled
          for (int i = 0; uses > 0 && i < (1 << 16) && !bar_try(&sh.full[s], (uses - 1) & 1); ++i) __nanosleep(64);
        }
    }
  } else {
    // ---- epilogue of all tiles but the CTA's last: a warp reaches the 32 lanes (rows) of its quarter
    const int et = tid - 32 * kDqWarps;
    auto epilogue_sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * kEpWarps) : "memory"); };
    auto any_failed = [&] {   // the same barrier, and one answer for all: a warp that left alone would strand the others at the next one
      uint32_t p;
      asm volatile(
          "{\n\t.reg .pred q, p;\n\t"
          "setp.ne.s32 q, %1, 0;\n\t"
          "bar.red.or.pred p, 1, %2, q;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(p)
          : "r"(*fail), "n"(32 * kEpWarps)
          : "memory");
      return p != 0;
    };
    int done = 0;
    if (MODE == RESIDUAL) {
      norm_top(nm, N, sh, et);
      epilogue_sync();
    }
    if (first < tiles) pdl_wait();   // Y may still be read by the kernel before this one; the norm's sums come from it or from earlier ones
#pragma unroll 1
    for (int tile = first; tile < tiles; tile += stride, ++done) {
      if (MODE != RESIDUAL && nm.ss_in) {
        const int t0 = (tile / feat_tiles) * nt;
        for (int i = et; i < nt; i += 32 * kEpWarps) {
          if (MODE == ROPE) token_pos[i] = __ldg(rp.pos + min(t0 + i, T - 1));
          token_fac[i] = t0 + i < T ? token_factor(nm, t0 + i) : 0.f;
        }
        epilogue_sync();
      }
      const bool ok = __all_sync(0xffffffffu, bar_wait<128>(&sh.acc_full, done & 1, fail, WAIT_EP));
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (tile + stride >= tiles) break;
      if (ok) park_tile(tmem, warp & 3, lane, rows, 0, 32, nt, fac);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      if (any_failed()) break;   // otherwise the tile is complete: a warp that gave up has raised the flag before
      if (lane == 0) bar_arrive_cluster(in_cta(sa(&sh.acc_empty), lead));
      const int t0 = (tile / feat_tiles) * nt, row0 = (tile % feat_tiles) * 256 + side * 128;
      if (MODE == RESIDUAL) store_residual(rows, nm, norm_scale(sh), T, N, t0, row0, nt, et, 32 * kEpWarps);
      else if (MODE == ROPE) store_rope(rows, rp, token_pos, Y, T, N, t0, row0, nt, et, 32 * kEpWarps);
      else store_tile<MODE == GATED>(rows, Y, T, N, t0, row0, nt, et, 32 * kEpWarps);
      epilogue_sync();   // `rows` is free for the next tile
    }
  }
  // ---- the CTA's last tile, by all warps: those that are not the epilogue's are idle by now
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const bool live = first < tiles && !*fail;
  const int last_tile = first < tiles ? first + (tiles - 1 - first) / stride * stride : 0;
  const int t_base = (last_tile / feat_tiles) * nt, row0 = (last_tile % feat_tiles) * 256 + side * 128;
  if (S == 1) {
    if (live && warp < 16) park_tile(tmem, warp & 3, lane, rows, 32 * (warp >> 2), 128, nt, fac);
    __syncthreads();
    if (live) {
      pdl_wait();
      if (MODE == RESIDUAL) store_residual(rows, nm, norm_scale(sh), T, N, t_base, row0, nt, tid, kThreads);
      else if (MODE == ROPE) store_rope(rows, rp, token_pos, Y, T, N, t_base, row0, nt, tid, kThreads);
      else store_tile<MODE == GATED>(rows, Y, T, N, t_base, row0, nt, tid, kThreads);
    }
  } else {
    // The split tile meets in the CTA that finishes a token: CTA (split, side) does tokens [split nt / S, (split + 1) nt / S) of its side's
    // rows. Every CTA writes its fp32 partials there, P[split][token][128 rows], and reads only its own shared memory afterwards: one
    // cluster barrier. (Partials parked locally and fetched by the finishing CTA: a round trip of distributed shared memory and a second
    // barrier more, 1.5 us a launch at 96 tokens.) Where P does not fit beside the stages it lies over them: then all CTAs' MMAs have
    // to be done first.
    const int chunk = nt / S;
    float* P = reinterpret_cast<float*>(base + (p_apart ? ns * stage_bytes : 0));
    if (!p_apart) cluster_barrier();
    if (live && warp < 16) {
#pragma unroll 1
      for (int c = 8 * (warp >> 2); c < nt; c += 32) {
        uint32_t v[8];
        tmem_ld8(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + c, v);
        const int owner = c / chunk;
        const uint32_t to = in_cta(sa(P + (size_t)(split * chunk + c - owner * chunk) * 128 + 32 * (warp & 3) + lane), 2 * owner + side);
#pragma unroll
        for (int j = 0; j < 8; ++j) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(to + 512 * j), "r"(v[j]) : "memory");
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    cluster_barrier();   // every CTA's partials are there, and nobody writes here any more
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (live) pdl_wait();
    constexpr int kWarps = kThreads / 32;
    uint2 next = make_uint2(0u, 0u), w4 = next;   // RESIDUAL: this lane's four columns of the next token's row, and of the norm's weight
    auto fetch = [&](int k) {
      const int t = t_base + split * chunk + k;
      if (MODE == RESIDUAL && k < chunk && t < T && row0 < N) next = *reinterpret_cast<const uint2*>(nm.x + (size_t)t * N + row0 + 4 * lane);
    };
    const float p = MODE == RESIDUAL ? norm_scale(sh) : 1.f, scale = 1.f / p;
    if (MODE == RESIDUAL && live) {
      if (row0 < N) w4 = __ldg(reinterpret_cast<const uint2*>(nm.w + row0 + 4 * lane));
      fetch(warp);
    }
    for (int k = warp; live && k < chunk; k += kWarps) {
      const int t = t_base + split * chunk + k;
      if (t >= T) break;
      const uint2 r = next;
      fetch(k + kWarps);
      float4 v[kMaxSplit];   // sum in split order, four rows a lane
#pragma unroll
      for (int s = 0; s < kMaxSplit; ++s)
        if (s < S) v[s] = reinterpret_cast<const float4*>(P + (size_t)(s * chunk + k) * 128)[lane];
      float4 a = v[0];
#pragma unroll
      for (int s = 1; s < kMaxSplit; ++s)
        if (s < S) a.x += v[s].x, a.y += v[s].y, a.z += v[s].z, a.w += v[s].w;
      const float f = fac ? token_fac[split * chunk + k] : 1.f;
      half2 h01 = __floats2half2_rn(a.x * f, a.y * f), h23 = __floats2half2_rn(a.z * f, a.w * f);
      if (MODE == ROPE) {   // as store_rope; the lane's four columns are all in one half of a head
        const int d2 = rp.D >> 1, row = row0 + 4 * lane, head = row / rp.D, in_head = row - head * rp.D, local = in_head & (d2 - 1);
        const uint32_t p01 = __shfl_xor_sync(0xffffffffu, as_u32(h01), d2 >> 2), p23 = __shfl_xor_sync(0xffffffffu, as_u32(h23), d2 >> 2);
        if (head >= rp.n_q + 2 * rp.n_kv) continue;
        const int pos = token_pos[split * chunk + k];
        if (head < rp.n_q + rp.n_kv) {
          const float4 c = __ldg(reinterpret_cast<const float4*>(rp.cos_t + (size_t)pos * d2 + local));
          float4 s = __ldg(reinterpret_cast<const float4*>(rp.sin_t + (size_t)pos * d2 + local));
          if (in_head < d2) s.x = -s.x, s.y = -s.y, s.z = -s.z, s.w = -s.w;
          const float2 a01 = __half22float2(h01), a23 = __half22float2(h23), b01 = __half22float2(as_h2(p01)), b23 = __half22float2(as_h2(p23));
          h01 = __floats2half2_rn(a01.x * c.x + b01.x * s.x, a01.y * c.y + b01.y * s.y);
          h23 = __floats2half2_rn(a23.x * c.z + b23.x * s.z, a23.y * c.w + b23.y * s.w);
        }
        const int page = head < rp.n_q ? 0 : __ldg(rp.bt + (pos >> rp.log2P));
        half* to = head_row(rp, Y, N, head, t, page, pos & ((1 << rp.log2P) - 1)) + in_head;
        *reinterpret_cast<uint2*>(to) = make_uint2(as_u32(h01), as_u32(h23));
        continue;
      }
      if (MODE == RESIDUAL) {   // as residual8
        if (row0 >= N) break;
        const size_t at = (size_t)t * N + row0 + 4 * lane;
        h01 = __hadd2(as_h2(r.x), h01), h23 = __hadd2(as_h2(r.y), h23);
        const float2 x01 = __half22float2(h01), x23 = __half22float2(h23), w01 = __half22float2(as_h2(w4.x)), w23 = __half22float2(as_h2(w4.y));
        *reinterpret_cast<uint2*>(nm.x + at) = make_uint2(as_u32(h01), as_u32(h23));
        *reinterpret_cast<uint2*>(nm.xw + at) = make_uint2(as_u32(__floats2half2_rn(x01.x * w01.x * scale, x01.y * w01.y * scale)),
                                                           as_u32(__floats2half2_rn(x23.x * w23.x * scale, x23.y * w23.y * scale)));
        const float ss = warp_sum(fmaf(x01.x, x01.x, fmaf(x01.y, x01.y, fmaf(x23.x, x23.x, x23.y * x23.y))));
        if (lane == 0) {
          nm.ss_out[(size_t)t * nm.parts + (row0 >> 7)] = ss;
          if (row0 == 0) nm.inv_out[t] = p;
        }
        continue;
      }
      half* y = Y + (size_t)t * N;
      if (MODE == GATED) {   // rows 16 k + 0..7 gates, 16 k + 8..15 their up rows: two lanes further on
        const uint32_t u01 = __shfl_xor_sync(0xffffffffu, as_u32(h01), 2), u23 = __shfl_xor_sync(0xffffffffu, as_u32(h23), 2);
        if ((lane & 2) == 0) {
          const int f = (row0 >> 1) + 8 * (lane >> 2) + 4 * (lane & 1);
          const half2 o01 = as_h2(gated2(as_u32(h01), u01)), o23 = as_h2(gated2(as_u32(h23), u23));
          const half o[4] = {__low2half(o01), __high2half(o01), __low2half(o23), __high2half(o23)};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (f + e < N) y[f + e] = o[e];
        }
      } else {
        const int f = row0 + 4 * lane;
        if (f + 3 < N && (N & 3) == 0) {
          *reinterpret_cast<uint2*>(y + f) = make_uint2(as_u32(h01), as_u32(h23));
        } else {
          const half o[4] = {__low2half(h01), __high2half(h01), __low2half(h23), __high2half(h23)};
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (f + e < N) y[f + e] = o[e];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (S == 1) cluster_barrier();   // the pair is done with its tensor memory and with each other's barriers (S > 1: since the barrier above)
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
  }
}

static int resident_clusters(int S, size_t smem) {   // clusters of 2 S CTAs the GPU holds at once; asked once per device
  static int known[kMaxDevices][kMaxSplit + 1] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  if (known[dev][S] == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2 * S, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(2 * S), cfg.blockDim = dim3(kThreads), cfg.dynamicSmemBytes = smem, cfg.attrs = attr, cfg.numAttrs = 1;
    int num = 0;
    if (cudaOccupancyMaxActiveClusters(&num, prefill_gemm_tiled_kernel<PLAIN>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      num = 0;
    }
    known[dev][S] = num > 0 ? num : -1;
  }
  return known[dev][S] > 0 ? known[dev][S] : 0;
}

cudaError_t prefill_gemm_tiled_status(int* code) {
  return cudaMemcpyFromSymbol(code, g_tiled_status, sizeof(int), 0, cudaMemcpyDeviceToHost);
}

// Y[T, N]; N = rows of W (swiglu: of outputs, W has 2 N rows in paired layout). force_split: 0, or the S to use.
cudaError_t prefill_gemm_tiled_dispatch(const void* Wt, const void* X, void* Y, int T, int N, int K, int swiglu, int force_split,
                                        const PrefillNorm* norm, const PrefillRope* rope, cudaStream_t st) {
  const int nunit = K / 128, row_tiles = swiglu ? (N + 7) / 8 : (N + 15) / 16, feat_tiles = (row_tiles + 15) / 16;
  auto bytes = [](int tokens, int stages, int per_token) { return 1024 + (size_t)tokens * (128 * stages + per_token); };
  const size_t smem_max = 224 * 1024;   // beside the static part
  static size_t allowed[4][kMaxDevices] = {};
  const int mode = rope ? ROPE : norm && norm->x ? RESIDUAL : swiglu ? GATED : PLAIN;
  if (mode == RESIDUAL && (swiglu || N % 128)) return cudaErrorInvalidValue;
  if (mode == ROPE && (swiglu || !norm || norm->x || (rope->D != 64 && rope->D != 128))) return cudaErrorInvalidValue;
  auto kern = mode == ROPE ? prefill_gemm_tiled_kernel<ROPE> : mode == RESIDUAL ? prefill_gemm_tiled_kernel<RESIDUAL>
              : mode == GATED ? prefill_gemm_tiled_kernel<GATED> : prefill_gemm_tiled_kernel<PLAIN>;
  cudaError_t e = allow_dynamic_smem(prefill_gemm_tiled_kernel<PLAIN>, smem_max, allowed[PLAIN]);   // resident_clusters asks for this one
  if (e == cudaSuccess && mode != PLAIN) e = allow_dynamic_smem(kern, smem_max, allowed[mode]);
  if (e != cudaSuccess) return e;
  // Tokens per tile (equal tiles, so that the last is not nearly empty; up to eight more of them than there have to be) and split of
  // K, by estimated time. In microseconds: a unit takes 0.35 (dequantization and issue) or, from 126 tokens on, 0.11 + 0.0019 a token (MMA and
  // activations with the chip full); beside that a launch takes 1.0 + 0.0162 a token where a pair works alone and 2.1 / 2.7 + 0.0206 a token
  // where 2 / 4 pairs exchange partial tiles; and up to 2.8 are lost with the SMs that the launch's last wave leaves none of to the start of the
  // next one. Measured on launches in a row of the four matrices of TinyLlama, 8B and 70B shapes, 16 .. 4096 tokens, every choice (3,570; plain and
  // SwiGLU epilogues): the pick is 0.2 % off the best on average, 6 % at worst (TinyLlama, down, 150 tokens). With a unit in proportion to its tokens
  // (0.00264) the pick was 0.75 % off and 14 % at worst: 128-token tiles in many waves looked cheap. Whole prompts, that unit / this one, us:
  // 70B shape (4 layers) 230 tokens 1,788 / 1,734, 256 1,853 / 1,771, 512 3,397 / 3,196, 1200 7,865 / 7,609; 8B shape (8 layers) 512 tokens
  // 1,815 / 1,882, 700 2,485 / 2,418, 1000 3,388 / 3,252; TinyLlama within 0.7 %, but 1200 and 2000 tokens 1 % faster.
  int S = 0, nt = 0, tiles = 0;
  double best = 0;
  const int least = (T + kMaxTokens - 1) / kMaxTokens;
  int least_split = 1;   // kMaxChain
  while (least_split < kMaxSplit && nunit > kMaxChain * least_split && resident_clusters(2 * least_split, smem_max) > 0) least_split *= 2;
  for (int c = force_split ? 1 : least_split; c <= kMaxSplit; c *= 2) {
    const int room = resident_clusters(c, smem_max);
    if (room == 0 || (force_split ? c != force_split : c > 1 && nunit / c < 2)) continue;
    const int units = (nunit + c - 1) / c;
    for (int ntt = least; ntt < least + 8; ++ntt) {
      const int n = ((T + ntt - 1) / ntt + 31) / 32 * 32, count = feat_tiles * ((T + n - 1) / n), waves = (count + room - 1) / room;
      const double unit = units * (n * 0.0019 + 0.11 > 0.35 ? n * 0.0019 + 0.11 : 0.35), fill = (double)(count - (waves - 1) * room) / room;   // of the last wave
      const double cost = (c == 1 ? 1.0 + 0.0162 * n + waves * (unit + 0.4) : waves * (1.45 + 0.32 * c + 0.0206 * n + unit)) +
                          2.8 * (fill < 0.36 ? 0 : fill > 0.86 ? 1 : 2 * (fill - 0.36));
      if (S == 0 || cost < best) best = cost, S = c, nt = n, tiles = count;
      if (n == 32) break;
    }
  }
  if (S == 0) return cudaErrorNotSupported;
  const int ns = nt <= 128 ? 6 : 4;   // what tensor memory has left beside the accumulator
  // beside the stages: the fp16 tile, or the fp32 partials of a split one where they fit
  const int p_apart = S > 1 && bytes(nt, ns, 512) <= smem_max;
  const size_t smem = bytes(nt, ns, S == 1 ? 256 : p_apart ? 512 : 0);
  const int room = resident_clusters(S, smem_max);
  CUtensorMap xmap;
  if (!encode_activation_map(&xmap, X, T, K, nt / 2, 2)) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * S, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(2 * S * (S > 1 || tiles < room ? tiles : room));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, xmap, (const uint8_t*)Wt, (half*)Y, T, N, row_tiles, nunit, nt, S, feat_tiles, tiles, ns, p_apart,
                            norm ? *norm : PrefillNorm{}, rope ? *rope : PrefillRope{});
}

}  // namespace b200
