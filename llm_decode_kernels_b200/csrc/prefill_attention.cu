// Attention of a prompt: T query tokens at positions start .. start + T - 1 over one sequence's paged cache (their own keys and
// values already appended), causal, grouped-query heads.
//
// The batched decode kernel (paged_attention.cu) treats every query token as a sequence of its own and reads the cache once per
// token: T^2 / 2 rows of K and V per kv head, 40 of the 74 ms of a 4096-token prompt. Here a block owns 128 query rows of one kv
// head - row = (token, head of the group), so the heads of a group share what is read - and walks over the context in tiles of 64
// tokens with an online softmax (FlashAttention, Dao et al. 2022), both contractions as mma.m16n8k16 out of a cp.async ring. Rows of
// 128 / 256 bytes are stored with their 16-byte pieces XOR-swizzled by the row, which keeps ldmatrix free of bank conflicts.
// Bound by the warp-level MMAs and the exponentials between them. Where a short prompt continues a long context the blocks are
// few: the context is then cut into splits of whole tiles, whose partials paged_attn_combine_kernel merges.
#include "common.cuh"
#include "prefill.h"
#include <math_constants.h>

namespace b200 {

namespace {

constexpr int kWarps = 8, kThreads = kWarps * 32, kRows = 16 * kWarps, kTile = 64;
template <int D> constexpr int stages() { return D == 64 ? 3 : 2; }
template <int D> constexpr size_t smem_bytes() { return (size_t)stages<D>() * 2 * kTile * D * sizeof(half); }

DEVI uint32_t sa(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
DEVI void cp16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
DEVI void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
DEVI void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
DEVI void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
DEVI float quad_max(float v) {
  v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
  return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
}
DEVI float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

}  // namespace

// Grid (row blocks, n_kv, splits). q rows: token t at q + t * q_stride, heads one after the other. PS tokens of context per split (a
// multiple of kTile). A row whose context lies in the first split writes `out`; others leave un-normalised partials.
template <int D>
__global__ void __launch_bounds__(kThreads, D == 64 ? 2 : 1)
prefill_attn_kernel(const half* __restrict__ q, int q_stride, const half* __restrict__ kc, const half* __restrict__ vc,
                    const int* __restrict__ bt, int start, int T, int n_kv, int log2hpg, int log2P, int PS, float sl2,
                    float* __restrict__ o_part, float* __restrict__ m_part, float* __restrict__ l_part, half* __restrict__ out) {
  constexpr int KS = D / 16, NB = D / 8, CH = D / 8, NS = stages<D>(), STAGE = 2 * kTile * D * 2;
  extern __shared__ __align__(128) uint8_t ring[];
  pdl_launch_dependents();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int hpg = 1 << log2hpg, n_q = n_kv << log2hpg, nsplit_max = gridDim.z;
  const int rb = gridDim.x - 1 - blockIdx.x;   // late tokens see the most context: they start first
  const int kvh = blockIdx.y, split = blockIdx.z, row0 = rb * kRows;
  const int last = start + min(T - 1, (row0 + kRows - 1) >> log2hpg);   // the block's last position
  const int k0 = split * PS, k1 = min(last + 1, k0 + PS);
  if (k0 >= k1) return;
  pdl_wait();

  const uint32_t ring_s = sa(ring);
  auto load = [&](int tile, int slot) {   // tokens k0 + 64 tile ..; past the block's context: its last token again (masked)
#pragma unroll
    for (int c = tid; c < kTile * CH; c += kThreads) {
      const int r = c / CH, ch = c % CH, j = min(k0 + tile * kTile + r, last);
      const size_t off = ((((size_t)__ldg(bt + (j >> log2P)) * n_kv + kvh) << log2P) + (j & ((1 << log2P) - 1))) * D + ch * 8;
      const uint32_t dst = ring_s + slot * STAGE + r * (2 * D) + ((ch ^ (r & 7)) << 4);
      cp16(dst, kc + off);
      cp16(dst + kTile * D * 2, vc + off);
    }
  };
  const int ntiles = (k1 - k0 + kTile - 1) / kTile;
#pragma unroll
  for (int i = 0; i < NS - 1; ++i) {
    if (i < ntiles) load(i, i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // this lane's two rows: g and g + 8 of the warp's sixteen
  int pos[2];
  const half* qp[2];
  size_t row_of[2];   // (token, query head) index
  bool live[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = row0 + warp * 16 + g + 8 * i, t = r >> log2hpg, h = (kvh << log2hpg) + (r & (hpg - 1));
    live[i] = t < T;
    const int tc = min(t, T - 1);
    pos[i] = start + tc;
    qp[i] = q + (size_t)tc * q_stride + (size_t)h * D;
    row_of[i] = (size_t)tc * n_q + h;
  }
  uint32_t qa[KS][4];
#pragma unroll
  for (int k = 0; k < KS; ++k) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      qa[k][i] = *reinterpret_cast<const uint32_t*>(qp[i] + 16 * k + 2 * t4);
      qa[k][2 + i] = *reinterpret_cast<const uint32_t*>(qp[i] + 16 * k + 8 + 2 * t4);
    }
  }
  const int wlast = start + min(T - 1, (row0 + warp * 16 + 15) >> log2hpg), wfirst = start + min(T - 1, (row0 + warp * 16) >> log2hpg);

  float m[2] = {-CUDART_INF_F, -CUDART_INF_F}, l[2] = {0.f, 0.f}, acc[NB][4];
#pragma unroll
  for (int n = 0; n < NB; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[n][e] = 0.f;

  const int mi = lane >> 3, lr = lane & 7;
#pragma unroll 1
  for (int it = 0; it < ntiles; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(NS - 2) : "memory");
    __syncthreads();   // tile `it` is there for everybody, and everybody is done with the slot that is filled next
    if (it + NS - 1 < ntiles) load(it + NS - 1, (it + NS - 1) % NS);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int j0 = k0 + it * kTile;
    if (j0 > wlast) continue;   // this warp's rows see none of it
    const uint32_t ks = ring_s + (it % NS) * STAGE, vs = ks + kTile * D * 2;
    float s[kTile / 8][4];
#pragma unroll
    for (int n = 0; n < kTile / 8; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
    for (int k = 0; k < KS; ++k)
#pragma unroll
      for (int n2 = 0; n2 < kTile / 16; ++n2) {
        uint32_t b[4];
        const int r = n2 * 16 + (mi >> 1) * 8 + lr, ch = 2 * k + (mi & 1);
        ldsm4(b, ks + r * (2 * D) + ((ch ^ (r & 7)) << 4));
        mma16816(s[2 * n2], qa[k], b[0], b[1]);
        mma16816(s[2 * n2 + 1], qa[k], b[2], b[3]);
      }
    if (j0 + kTile - 1 > wfirst) {   // the diagonal runs through this tile
#pragma unroll
      for (int n = 0; n < kTile / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j0 + 8 * n + 2 * t4 + (e & 1) > pos[e >> 1]) s[n][e] = -CUDART_INF_F;
    }
    float sub[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float mx = -CUDART_INF_F;
#pragma unroll
      for (int n = 0; n < kTile / 8; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * i], s[n][2 * i + 1]));
      const float mn = fmaxf(m[i], quad_max(mx) * sl2);   // log2 units
      sub[i] = mn == -CUDART_INF_F ? 0.f : mn;            // nothing visible yet: every probability is 2^-inf
      const float alpha = exp2f(m[i] - sub[i]);
      m[i] = mn;
      l[i] *= alpha;
#pragma unroll
      for (int n = 0; n < NB; ++n) acc[n][2 * i] *= alpha, acc[n][2 * i + 1] *= alpha;
    }
#pragma unroll
    for (int k = 0; k < kTile / 16; ++k) {
      uint32_t p[4];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float a = exp2f(fmaf(s[2 * k + h][2 * i], sl2, -sub[i])), b = exp2f(fmaf(s[2 * k + h][2 * i + 1], sl2, -sub[i]));
          l[i] += a + b;
          p[2 * h + i] = as_u32(__floats2half2_rn(a, b));
        }
#pragma unroll
      for (int d2 = 0; d2 < NB / 2; ++d2) {
        uint32_t b[4];
        const int r = k * 16 + (mi & 1) * 8 + lr, ch = 2 * d2 + (mi >> 1);
        ldsm4t(b, vs + r * (2 * D) + ((ch ^ (r & 7)) << 4));
        mma16816(acc[2 * d2], p, b[0], b[1]);
        mma16816(acc[2 * d2 + 1], p, b[2], b[3]);
      }
    }
  }

#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float L = quad_sum(l[i]);
    if (!live[i] || pos[i] < k0) continue;
    if (pos[i] < PS || nsplit_max == 1) {
      const float r = 1.f / L;
      half* o = out + row_of[i] * D + 2 * t4;
#pragma unroll
      for (int n = 0; n < NB; ++n)
        *reinterpret_cast<half2*>(o + 8 * n) = __floats2half2_rn(acc[n][2 * i] * r, acc[n][2 * i + 1] * r);
    } else {
      const size_t at = row_of[i] * nsplit_max + split;
      float* o = o_part + at * D + 2 * t4;
#pragma unroll
      for (int n = 0; n < NB; ++n) *reinterpret_cast<float2*>(o + 8 * n) = make_float2(acc[n][2 * i], acc[n][2 * i + 1]);
      if (t4 == 0) m_part[at] = m[i] * 0.69314718055994530942f, l_part[at] = L;   // natural-log units, as the combine step reads
    }
  }
}

// floats of scratch for `splits` partials
static size_t scratch_floats(int T, int n_q, int D, int splits) { return (size_t)T * n_q * splits * (D + 2); }

bool prefill_attention_takes(int D, int n_q, int n_kv) {
  const int hpg = n_q / n_kv;
  return (D == 64 || D == 128) && (hpg & (hpg - 1)) == 0 && hpg <= kRows;
}

// pos: the T positions on the device (read by the combine step). scratch may be null: one split then.
cudaError_t prefill_attention_dispatch(const void* q, int q_stride, const void* kc, const void* vc, const int* bt, const int* pos,
                                       int start, int T, int n_q, int n_kv, int D, int log2P, float* scratch, size_t scratch_len,
                                       void* out, cudaStream_t st) {
  const int hpg = n_q / n_kv;
  int log2hpg = 0;
  while ((1 << log2hpg) < hpg) ++log2hpg;
  const int row_blocks = (T * hpg + kRows - 1) / kRows, tiles = (start + T + kTile - 1) / kTile;
  // one wave of blocks (two per SM at head_dim 64), at least four tiles each so that a split outweighs its merge
  const int want = kNumSMs * (D == 64 ? 2 : 1);
  int splits = want / (row_blocks * n_kv);
  splits = splits < tiles / 4 ? splits : tiles / 4;
  while (splits > 1 && scratch_floats(T, n_q, D, splits) > scratch_len) --splits;
  if (splits < 1) splits = 1;
  const int PS = (tiles + splits - 1) / splits * kTile;
  splits = (start + T + PS - 1) / PS;
  float *o_part = scratch, *m_part = scratch + (size_t)T * n_q * splits * D, *l_part = m_part + (size_t)T * n_q * splits;
  const float sl2 = 1.44269504088896340736f / sqrtf((float)D);
  auto kern = D == 64 ? prefill_attn_kernel<64> : prefill_attn_kernel<128>;
  const size_t smem = D == 64 ? smem_bytes<64>() : smem_bytes<128>();
  static size_t allowed[2][kMaxDevices] = {};
  const cudaError_t e = allow_dynamic_smem(kern, smem, allowed[D == 128]);
  if (e != cudaSuccess) return e;
  B200_LAUNCH(kern, dim3(row_blocks, n_kv, splits), dim3(kThreads), smem, st, (const half*)q, q_stride, (const half*)kc,
              (const half*)vc, bt, start, T, n_kv, log2hpg, log2P, PS, sl2, o_part, m_part, l_part, (half*)out);
  if (splits > 1) return attention_combine_dispatch(o_part, m_part, l_part, pos, PS, splits, n_q, T, D, out, st);
  return cudaPeekAtLastError();
}

}  // namespace b200
