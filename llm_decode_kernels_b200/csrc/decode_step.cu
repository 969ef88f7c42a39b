// One persistent kernel for the whole batch-1 decode step (all layers, LM head, greedy argmax).
//
// Why: at TinyLlama size the step streams 0.55 GB of INT4 weights, 86 us at the B200's measured HBM bandwidth,
// while the same step as 225 separate launches (the reference's structure, runtime/model.py:216-233) costs ~900 us
// of launch and pipeline-drain latency. Here one CTA per SM stays resident for the whole step:
//
//   * a producer warp streams this CTA's row tiles of every weight matrix - and, on the CTAs that do attention, the
//     K/V pages of their head - in the order the step consumes them, into a shared-memory ring with 1-D bulk async
//     copies (cp.async.bulk + mbarrier transaction counts). Neither weights nor cached K/V depend on this step's
//     activations, so the producer runs ahead of the computation by the depth of the ring and HBM never idles
//     while CTAs wait for each other;
//   * 11 consumer warps do the arithmetic out of the ring on the tensor cores (see "inner product" below), with the
//     row length K split across the warps: warp w owns the 128-column units w, w + 11, ... of every row tile, so it
//     needs only its own 128-element pieces of the activation vector and fetches exactly those - no CTA-wide staging
//     pass and no barrier in front of a GEMV. The warps' partial sums meet in shared memory once per matrix.
//     (Twelve warps in all, three per scheduler: a thread then has 168 registers, and this kernel must not spill -
//     with 227 KB of the SM's memory configured as shared there is next to no L1 left, so spilled registers would
//     be fetched from the L2, a microsecond each time, in a kernel whose phases last a microsecond. A thirteenth
//     warp puts four on one scheduler and caps every thread at 128 registers, seventeen warps at 96;)
//   * CTAs exchange activation vectors through global memory WITHOUT grid barriers: every fp16 result is stored
//     as a 32-bit word (tag << 16 | value) whose tag is this step's epoch; a consumer polls the words it needs until
//     all carry the current tag. One store + one load crosses the chip instead of fence + atomic + poll + load.
//     Every CTA keeps its own copy of the residual stream in shared memory (each warp its own units of it) and redoes
//     the (tiny) residual add and RMSNorm, so those never touch global memory.
//
// Weights are read from the tile layout of the tensor-core GEMV (gemv_tile_repack_kernel in gemv_w4a16.cu): per
// 16-row tile and 128-column unit one 1088-byte block, tiles back to back. A CTA owns a contiguous range of tiles of
// each matrix, so its share is one contiguous byte range and a ring stage is ONE bulk copy of up to `ups` blocks.
// The gate|up matrix uses the paired form of the layout (gate row i and up row i in one tile), which puts both
// halves of a SwiGLU output into the same thread.
//
// Inner product on the integer tensor cores. (word & 0x0F0F0F0F) and ((word >> 4) & 0x0F0F0F0F) are registers of four
// unsigned-byte weights each - three integer instructions for 8 weights - so a 16-row x 128-column block of W is
// four mma.m16n8k32 (u8 x s8 -> s32). The activations go in as 15-bit fixed point: staging scales a unit's x by
// 2^s (s from the unit's max|x|; a unit belongs to one warp, so this costs five shuffles and no reduction over the
// CTA), rounds to an integer X, |X| < 2^14, and splits it into two signed byte digits, X = 256 hi + lo. The digits
// ride in columns 0 and 1 of the B operand, which a batch-1 GEMV leaves idle anyway, the accumulation is exact, and
//     sum_k (q_k - z) * scale * x_k  =  scale * (2^-s * (256 C[.][0] + C[.][1]) - z * sum_k x_k)        per unit.
// Rounding x to 2^-14 of its unit's maximum is finer than the fp16 rounding x already carries, except for elements
// far below the maximum, whose absolute error it bounds by 2^-15 of the maximum (normwise ~1e-5 on the output).
// A NaN or infinity in a unit of x - which an integer cannot carry - turns that unit's factor 2^-s into NaN, so
// every row's output is NaN as in the reference.
// Why this form: a GEMV phase of this kernel is bound by instruction issue, and most instructions around the
// weights (LOP3, SHF, HFMA2) issue at half rate. Measured per tile-unit and warp, eight warps per SM: masked nibbles
// as fp16 subnormals into mma.m16n8k16, 5 integer instructions + 1 MMA per 8 weights of a row pair: 320 cycles; the
// same masks into half2 FMAs: 306; this form, 3 integer instructions per 8 weights and 4 MMAs per tile-unit: 195.
// (The e4m3 MMA of the same shape would fit too - a nibble in the low half of an e4m3 byte is exactly q * 2^-9 -
// but it is emulated on this part: 385.)
// The per-element weight this stands for is the format's dequantized weight (dequant_w4a16 in gemv_w4a16.cu proves
// the format bit-exactly).
//
// Phases per layer (the reference's operator order and the rounding points of its fused kernels, but for the
// normalised row, which is not rounded to fp16 before the product):
//   A  resid += down[l-1] (layer 0: resid = embedding row);  x = RMSNorm(resid) * ln1;  qkv = Wqkv x
//   B  attention: RoPE on q and k, append k, v to the paged cache, online softmax over the cached tokens (from the ring).
//      Short contexts: one CTA per query head. Longer ones, with an exchange of its own (the wide one): a CTA takes one kv head and
//      one slice of the context for ALL query heads of the group (up to 8), so every cached row is copied and read once,
//      both contractions as warp-level MMAs; one CTA per head merges the slices' outputs. (TinyLlama shape at 8192
//      cached tokens: 695 us a token with up to four CTAs per query head, 440 this way.) Without: see att_plan.
//   C  o = Wo attn
//   D  resid += o;  x = RMSNorm(resid) * ln2;  act = SwiGLU(Wgate x, Wup x)
//   E  down = Wdown act
// then resid += down;  x = RMSNorm(resid) * norm_f;  logits = Whead x;  per-CTA argmax candidates; CTA 0 merges
// them (lowest index wins ties), writes tok, history[pos], pos + 1 and the new epoch.
// The norm's factor rsqrt(mean(resid^2) + eps) multiplies the outputs of the GEMV behind it (x is staged as resid * ln).
// One barrier over the consumer threads per phase, between the warps' partial sums (and sums of squares) and the threads that
// add them up; the partial-sum buffer alternates between phases so that no second one is needed.
// The code of the loop is kept small - one copy of what serves several phases, loops not unrolled where nothing is gained:
// at 101 KB the fetches of 90 to 180 lines per layer and SM from the L2 were 12 us of a token, at 85 KB there are none.
//
// Every wait (mbarrier or tag poll) is bounded. A wait that runs out records a code in StepCtrl::error, raises an
// abort flag that all later waits honour at once, and the CTA leaves after its copies in flight have landed; the
// host reads the code after the step. Nothing here can spin forever.
#include "common.cuh"
#include "decode_step.h"
#include <math_constants.h>

namespace b200 {

namespace {

#ifndef B200_STEP_CONSUMER_WARPS
#define B200_STEP_CONSUMER_WARPS 11   // build-time knob for measurements
#endif
constexpr int kNCW = B200_STEP_CONSUMER_WARPS;   // consumer warps (with the producer: 12 warps = 3 per scheduler, 168 registers)
constexpr int kNT = kNCW * 32;              // consumer threads
constexpr int kThreads = kNT + 32;          // + producer warp
constexpr int kMaxStages = 16;
constexpr int kSpinLimit = 1 << 18;         // polls / try_waits before a wait gives up (tens of milliseconds)
constexpr int kHeaderBytes = 2048;
constexpr int kMaxKvTokens = 128;           // cached tokens per ring stage in attention (3 rounds of 11 warps x 4 tokens)
constexpr int kKvRounds = (kMaxKvTokens + 4 * kNCW - 1) / (4 * kNCW);
// Units of a row a warp polls and stages together: two, so that nothing spills, where a row is a few units per warp; more for long
// rows, which are bound by these trips to the L2 (28672 weights: 20 units per warp; 8 layers of the 70B shape 884 -> 858 us).
// Six or eight at a time spill and lose again.
constexpr int kBatch = 2, kBatchNorm = 2, kWideBatch = 4, kWideBatchNorm = 3;
constexpr int kWideUnits = 4;               // units per warp above which a row counts as long

enum : int { ERR_POLL = 1, ERR_FULL = 2, ERR_EMPTY = 3, ERR_TOKEN = 4 };

// ---- PTX wrappers --------------------------------------------------------------------------------------------
DEVI uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
DEVI void mbar_init(uint64_t* b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count));
}
DEVI void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
DEVI void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
DEVI bool mbar_try_wait(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
DEVI void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
DEVI void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kNT) : "memory"); }
// Barrier over the consumer threads that also ORs a flag: every thread gets the same answer, so the decision to
// leave the kernel is taken by all consumer threads together (a thread that left alone would strand the others
// at the next barrier).
DEVI bool consumer_sync_or(int flag) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.s32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(flag), "n"(kNT)
      : "memory");
  return r != 0;
}
DEVI uint4 ld_poll4(const uint32_t* p) {
  uint4 r;
  asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
  return r;
}
DEVI void st_tagged(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

DEVI void st_tagged2(uint32_t* p, uint32_t a, uint32_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(a), "r"(b) : "memory");
}

// ---- shared state of one CTA -----------------------------------------------------------------------------------
// Shared memory: [0, 128) full barriers, [128, 256) empty barriers, 256 abort flag, 272 sum scratch, 512 slices, 640 plan of
// the attention, 704 argmax keys, 1024 RoPE factors;
// from kHeaderBytes on: residual stream, then the areas whose offsets the host put into StepParams (off_*).
// Pointers into it are formed where they are used (one add of a kernel parameter) instead of being carried in
// registers through the whole step.
// How a step's attention is cut: A slices of `per` cached tokens. two: per kv head, the partials merged by one CTA per head, which
// publishes the attention output; staged: per query head, merged by the CTAs that stage it; neither: one CTA per query head.
// units: attention units of a layer, dealt to the CTAs in turn.
struct AttPlan { int A, per, two, staged, refresh, pos, units; };

// The shared memory is named where it is used and not carried as a pointer: a pointer that passes through a function or an asm
// statement loses its address space, and every access through it becomes a generic one.
extern __shared__ __align__(128) uint8_t step_smem[];
struct Cta {
  const StepParams* p;   // the kernel's parameter block (constant bank)
  uint32_t tagw;         // (tag << 16)
#ifdef B200_STEP_TRACE
  long long* tr;         // this CTA's row of the trace array (thread 0 stamps), or null
#endif
  DEVI uint64_t* full(int i) const { return reinterpret_cast<uint64_t*>(step_smem) + i; }
  DEVI uint64_t* empty(int i) const { return reinterpret_cast<uint64_t*>(step_smem) + kMaxStages + i; }
  DEVI volatile int* abort() const { return reinterpret_cast<volatile int*>(step_smem + 2 * kMaxStages * 8); }
  // kNCW floats: the warps' shares of sum(resid^2)
  DEVI float* red() const { return reinterpret_cast<float*>(step_smem + 2 * kMaxStages * 8 + 16); }
  // [H] residual stream, private copy of the CTA; unit u belongs to warp u % kNCW
  DEVI half* resid() const { return reinterpret_cast<half*>(step_smem + kHeaderBytes); }
  // activations of the running GEMV as byte-digit B fragments, 256 bytes per unit; unit u is written and read by one warp only
  DEVI half* xin() const { return reinterpret_cast<half*>(step_smem + p->off_xin); }
  DEVI float* xsum() const { return reinterpret_cast<float*>(step_smem + p->off_xsum); }   // [Kmax / 128][2] sum, 2^-s
  DEVI uint8_t* att() const { return step_smem + p->off_att; }                             // attention scratch (att_layout)
  DEVI const AttPlan& plan() const { return *reinterpret_cast<const AttPlan*>(step_smem + 640); }
  DEVI unsigned long long* keys() const { return reinterpret_cast<unsigned long long*>(step_smem + 704); }   // [2 kNCW]
  DEVI float* rope() const { return reinterpret_cast<float*>(step_smem + 1024); }          // [D/2] cos, [D/2] sin, page of pos
  // partial dot products, [warp][row slot], two buffers used by alternate phases
  DEVI float* part() const { return reinterpret_cast<float*>(step_smem + p->off_part); }
  DEVI uint8_t* stage(int slot) const { return step_smem + p->off_ring + (size_t)slot * p->stage_bytes; }
  DEVI StepCtrl* ctrl() const { return p->ctrl; }
  DEVI const StepLayer& layer(int l) const { return reinterpret_cast<const StepLayer*>(step_smem + p->off_table)[l]; }
};

// Phase stamps of the instrumented build (-DB200_STEP_TRACE): thread 0 of the CTA stores the nanosecond timer at slot
// `at` of the CTA's trace row. The normal build compiles these calls to nothing.
#ifdef B200_STEP_TRACE
DEVI void stamp(const Cta& c, int at) {
  if (c.tr && threadIdx.x == 0) {
    long long t_;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));
    c.tr[at] = t_;
  }
}
#else
DEVI void stamp(const Cta&, int) {}
#endif
#ifdef B200_STEP_TRACE
DEVI long long now_ns() {
  long long t_;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));
  return t_;
}
// slot `at` <- a duration (ns) instead of a time
DEVI void stamp_value(const Cta& c, int at, long long v) {
  if (c.tr && threadIdx.x == 0) c.tr[at] = v;
}
#else
DEVI void stamp_value(const Cta&, int, long long) {}
#endif
constexpr int kTraceHead = 8, kTracePerPhase = 5, kTraceAttn = 5, kTracePerLayer = 4 * kTracePerPhase + kTraceAttn;

DEVI void raise(const Cta& c, int code) {
  if (!*c.abort()) {
    *c.abort() = 1;
    atomicCAS(&c.ctrl()->error, 0, code);
    c.ctrl()->abort = 1;
  }
}

// Wait for a ring barrier phase. Returns false (and raises) if the bound is hit or the step is already aborting.
// `nap` nanoseconds of sleep follow every failed attempt: a waiting warp must not eat the issue slots of the warps
// it shares a scheduler with (the producer waits for most of the step).
DEVI bool wait_bar(const Cta& c, uint64_t* bar, uint32_t parity, int code, unsigned nap = 0) {
#pragma unroll 1
  for (int i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*c.abort()) return false;
    if (nap) __nanosleep(nap);
  }
  raise(c, code);
  return false;
}

// Consumer side of a ring stage; a build under trace adds to `waited` what it took.
DEVI bool wait_full(const Cta& c, int slot, uint32_t parity, long long& waited) {
#ifdef B200_STEP_TRACE
  const long long w0 = now_ns();
  const bool ok = wait_bar(c, c.full(slot), parity, ERR_FULL);
  waited += now_ns() - w0;
  return ok;
#else
  return wait_bar(c, c.full(slot), parity, ERR_FULL);
#endif
}

// ---- tagged exchange words -----------------------------------------------------------------------------------------
// A word of step s carries tag (s mod 65535) + 1, so a word left over from step s - 65535 would pass for a fresh one.
// That cannot happen: the output rows of every phase of every layer and the argmax candidates are rewritten in every
// step, and the partials of attention slices, of which a short context uses only a few, at least in every 1024th step
// (refresh_partials).
DEVI bool tags_ok(const Cta& c, uint4 v) {
  return ((((v.x ^ c.tagw) | (v.y ^ c.tagw) | (v.z ^ c.tagw) | (v.w ^ c.tagw)) >> 16) == 0);
}
DEVI uint2 payload(uint4 v) { return make_uint2((v.x & 0xFFFFu) | (v.y << 16), (v.z & 0xFFFFu) | (v.w << 16)); }

// Poll nb (<= NB, warp-uniform) granules of 4 tagged words, `stride` words apart, until all carry this
// step's tag; all loads of a round are in flight together. out[k] = the 4 fp16 payloads of granule k as 2 x half2.
template <int NB>
DEVI void poll_many(const Cta& c, const uint32_t* base, int stride, int nb, uint2 (&out)[NB]) {
  uint4 v[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k < nb) v[k] = ld_poll4(base + k * stride);
  int spins = 0;
#pragma unroll 1
  for (;;) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NB; ++k)
      if (k < nb && !tags_ok(c, v[k])) ok = false;
    if (ok || *c.abort()) break;
    if (++spins > kSpinLimit) { raise(c, ERR_POLL); break; }
    if ((spins & 255) == 0 && ((volatile StepCtrl*)c.ctrl())->abort) { *c.abort() = 1; break; }
#pragma unroll
    for (int k = 0; k < NB; ++k)
      if (k < nb && !tags_ok(c, v[k])) v[k] = ld_poll4(base + k * stride);
  }
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if (k < nb) out[k] = payload(v[k]);
}
DEVI uint2 poll4(const Cta& c, const uint32_t* p) {
  uint2 out[1];
  poll_many<1>(c, p, 0, 1, out);
  return out[0];
}
// The same for granules at unrelated places: entry k is at word offset off[k] from `base` (32-bit offsets: a dozen
// 64-bit pointers would not fit beside a dozen granules in flight); bit k of `mask` says whether entry k is in use
// (warp-uniform).
template <int NB>
DEVI void poll_list(const Cta& c, const uint32_t* base, const uint32_t (&off)[NB], uint32_t mask, uint2 (&out)[NB]) {
  uint4 v[NB];
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if ((mask >> k) & 1u) v[k] = ld_poll4(base + off[k]);
  int spins = 0;
#pragma unroll 1
  for (;;) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NB; ++k)
      if (((mask >> k) & 1u) && !tags_ok(c, v[k])) ok = false;
    if (ok || *c.abort()) break;
    if (++spins > kSpinLimit) { raise(c, ERR_POLL); break; }
    if ((spins & 255) == 0 && ((volatile StepCtrl*)c.ctrl())->abort) { *c.abort() = 1; break; }
#pragma unroll
    for (int k = 0; k < NB; ++k)
      if (((mask >> k) & 1u) && !tags_ok(c, v[k])) v[k] = ld_poll4(base + off[k]);
  }
#pragma unroll
  for (int k = 0; k < NB; ++k)
    if ((mask >> k) & 1u) out[k] = payload(v[k]);
}

// ---- x staging, per warp ------------------------------------------------------------------------------------------
// Warp w stages the units w, w + kNCW, ... of the activation vector: lane l holds granule l (4 values) of a unit.
// A unit's x goes to shared memory as the B fragments of the integer MMAs: X = round(x * 2^s), split into the signed
// byte digits hi and lo (X = 256 hi + lo, both in [-128, 127]), laid out as
//     xin words [unit][digit n = 0 (hi), 1 (lo)][t = 0..3][MMA m = 0..3][register r = 0..1]
// where lane (n, t) of tile_unit() loads its eight registers with two 16-byte reads. Register r of MMA m pairs with
// word 2 (m / 2) + r of the lane's four weight words, low nibbles (m even: elements e0 e4 e1 e5 of the word, in
// byte order) or high nibbles (m odd: e2 e6 e3 e7). Granule l = 4 elements of word (l % 8) / 2: elements e0..e3 on
// even lanes, e4..e7 on odd ones, so a lane pair swaps its packed bytes once and each lane permutes one register.
// xsum[2 u] = 2^-s sum X (for the zero-point term), xsum[2 u + 1] = 2^-s (both NaN if the unit is not finite).
DEVI void put_unit(const Cta& c, int u, float4 v, int lane) {
  // max|x| of the unit from the bit patterns (the order of non-negative floats is the order of their bits; NaN is above all)
  const uint32_t mx = __reduce_max_sync(0xffffffffu, max(max(__float_as_uint(v.x) & 0x7FFFFFFFu, __float_as_uint(v.y) & 0x7FFFFFFFu),
                                                         max(__float_as_uint(v.z) & 0x7FFFFFFFu, __float_as_uint(v.w) & 0x7FFFFFFFu)));
  const bool finite = mx < 0x7F800000u;                   // no infinity, no NaN
  const int e = max((int)(mx >> 23), 14);                 // exponent field: max|x| in [2^(e-127), 2^(e-126))
  const float sc = __int_as_float((267 - e) << 23);       // 2^s, s = 140 - e: 2^s max|x| in [2^13, 2^14)
  // round(x * 2^s) + 128 in the low bits of a float: adding 1.5 * 2^23 + 128 rounds to an integer (nearest even)
  // and leaves it, in two's complement, in the mantissa. Byte 0 of that, with its top bit flipped, is the lo digit
  // (X & 255 read as a signed byte), byte 1 is the hi digit ((X + 128) >> 8).
  constexpr float kMagic = 12582912.f + 128.f;
  const uint32_t w0 = __float_as_uint(fmaf(v.x, sc, kMagic)), w1 = __float_as_uint(fmaf(v.y, sc, kMagic));
  const uint32_t w2 = __float_as_uint(fmaf(v.z, sc, kMagic)), w3 = __float_as_uint(fmaf(v.w, sc, kMagic));
  const uint32_t kM = __float_as_uint(kMagic);            // w - kM = X
  const int xsum_i = __reduce_add_sync(0xffffffffu, (int)(w0 - kM) + (int)(w1 - kM) + (int)(w2 - kM) + (int)(w3 - kM));
  const float resc = finite ? __int_as_float((e - 13) << 23) : __int_as_float(0x7fc00000);   // 2^-s, or NaN
  if (lane == 0) {
    c.xsum()[2 * u] = (float)xsum_i * resc;               // the sum of what the MMAs multiply, rescaled
    c.xsum()[2 * u + 1] = resc;
  }
  // bytes: this granule's 4 elements in order
  const uint32_t lo = __byte_perm(__byte_perm(w0, w1, 0x0040), __byte_perm(w2, w3, 0x0040), 0x5410) ^ 0x80808080u;
  const uint32_t hi = __byte_perm(__byte_perm(w0, w1, 0x0051), __byte_perm(w2, w3, 0x0051), 0x5410);
  const int t = lane >> 3, wd = (lane & 7) >> 1, odd = lane & 1;
  uint32_t* dst = reinterpret_cast<uint32_t*>(c.xin()) + (size_t)u * 64 + t * 8 + ((wd >> 1) * 2 + odd) * 2 + (wd & 1);
  const uint32_t hi_o = __shfl_xor_sync(0xffffffffu, hi, 1), lo_o = __shfl_xor_sync(0xffffffffu, lo, 1);
  // even lane (e0..e3; partner e4..e7): low-nibble register (e0 e4 e1 e5); odd lane: high-nibble one (e2 e6 e3 e7)
  dst[0] = odd ? __byte_perm(hi, hi_o, 0x3726) : __byte_perm(hi, hi_o, 0x5140);
  dst[32] = odd ? __byte_perm(lo, lo_o, 0x3726) : __byte_perm(lo, lo_o, 0x5140);
}

// x <- E[0..K) (tagged).
template <int PB>
DEVI void stage_plain(const Cta& c, const uint32_t* E, int K, int warp, int lane) {
  const int nunit = K >> 7;
#pragma unroll 1
  for (int u0 = warp; u0 < nunit; u0 += kNCW * PB) {
    const int nb = min(PB, (nunit - u0 + kNCW - 1) / kNCW);
    uint2 v[PB];
    poll_many(c, E + 128 * u0 + 4 * lane, 128 * kNCW, nb, v);
#pragma unroll
    for (int k = 0; k < PB; ++k)
      if (k < nb) {
        const float2 a = __half22float2(as_h2(v[k].x)), b = __half22float2(as_h2(v[k].y));
        put_unit(c, u0 + kNCW * k, make_float4(a.x, a.y, b.x, b.y), lane);
      }
  }
  __syncwarp();
}

// resid <- resid + delta (delta tagged; or resid <- emb row when E == nullptr), x <- w * resid, and the warp's share of sum(resid^2).
// The factor rsqrt(mean(resid^2) + eps) of the norm is common to the whole row: it is applied to the outputs (reduce_emit), behind
// the barrier that is there anyway, and no warp waits for the others here. Waiting cost 0.4 us per norm, 19 us per token.
template <int NB>
DEVI void stage_norm(const Cta& c, const uint32_t* E, const half* emb_row, const half* w, int H, int warp, int lane) {
  const int nunit = H >> 7;
  uint2* rs = reinterpret_cast<uint2*>(c.resid());
  const uint2* wg = reinterpret_cast<const uint2*>(w);
  float ss = 0.f;
#pragma unroll 1
  for (int u0 = warp; u0 < nunit; u0 += kNCW * NB) {
    const int nb = min(NB, (nunit - u0 + kNCW - 1) / kNCW);
    uint2 d[NB], wv[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k)   // the norm weights travel while the residual is polled
      if (k < nb) wv[k] = __ldg(wg + 32 * (u0 + kNCW * k) + lane);
    if (E) poll_many(c, E + 128 * u0 + 4 * lane, 128 * kNCW, nb, d);
    float4 x[NB];
    float sq = 0.f;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      if (k < nb) {
        const int idx = 32 * (u0 + kNCW * k) + lane;
        uint2 r;
        if (E) {
          r = rs[idx];
          r.x = as_u32(__hadd2(as_h2(r.x), as_h2(d[k].x)));
          r.y = as_u32(__hadd2(as_h2(r.y), as_h2(d[k].y)));
        } else {
          r = __ldg(reinterpret_cast<const uint2*>(emb_row) + idx);
        }
        rs[idx] = r;
        const float2 a = __half22float2(as_h2(r.x)), b = __half22float2(as_h2(r.y));
        sq = fmaf(a.x, a.x, fmaf(a.y, a.y, fmaf(b.x, b.x, fmaf(b.y, b.y, sq))));
        const float2 wa = __half22float2(as_h2(wv[k].x)), wb = __half22float2(as_h2(wv[k].y));
        x[k] = make_float4(a.x * wa.x, a.y * wa.y, b.x * wb.x, b.y * wb.y);
      }
    }
    ss += warp_sum(sq);   // its shuffles fill the gaps in put_unit's chain
    put_unit(c, u0, x[0], lane);
#pragma unroll
    for (int k = 1; k < NB; ++k)
      if (k < nb) put_unit(c, u0 + kNCW * k, x[k], lane);
  }
  if (lane == 0) c.red()[warp] = ss;
  __syncwarp();
}
// the factor of the norm, behind a barrier after stage_norm
DEVI float norm_factor(const Cta& c, int H, float eps) {
  float v[kNCW];
#pragma unroll
  for (int k = 0; k < kNCW; ++k) v[k] = c.red()[k];
#pragma unroll
  for (int k = 0; k + 1 < kNCW; k += 2) v[k] += v[k + 1];
  float tot = v[0];
#pragma unroll
  for (int k = 2; k < kNCW; k += 2) tot += v[k];
  return rsqrtf(tot / (float)H + eps);
}

// ---- GEMV phase -----------------------------------------------------------------------------------------------------
// A weight matrix in tile layout. N = outputs (for gate|up: I, each output made of a gate and an up row).
struct Mat {
  const uint8_t* base;
  int N, K;
  int paired;          // 1: gate|up tiles (8 gate rows + their 8 up rows)
};

// This CTA's tiles [t0, t0 + nt) of a matrix, in ring stages of `ups` blocks: as many as a stage holds, but
//  - rows of which a stage holds two and more (up to 16 units): whole tiles, `whole` of them, and the loop over tiles in gemv. us a token of 8 layers
//    in the general loop / this one: 1280 columns (stages of 30) 138 / 133, 1536 (24) 144 / 139. One tile a stage leaves too much of the ring empty: 2560
//    columns 168 / 170, 2816 174.0 / 174.6;
//  - one tile of a row that fills more than a stage and no more than two passes of two units a warp (33 to 44 units): two stages of
//    22 at most, which are those two passes; 32 and the rest are three. 8 layers of 2048 columns, down's rows 4352 / 4608 / 5120 / 5504 / 5632:
//    122.0 / 120.5 / 122.1 / 123.0 / 124.0 -> 119.0 / 118.7 / 119.9 / 121.3 / 122.7. Not with more tiles, which want the ring full: 4096 columns, two
//    tiles of 5632 104.9 -> 105.3; 5120 columns (three and four tiles a matrix) 144.7 -> 151.6.
struct Slice { int t0, nt, ups, whole; };

// Position in the ring. Stages are used strictly in order by producer and consumers alike, so a slot index and a
// parity bit that flips on wrap-around replace a stage counter (and the divisions by the ring size it would need).
struct RingPos {
  int slot;
  uint32_t parity;
};
struct ProducerPos : RingPos {
  int count;   // stages passed (the abort path needs it)
};
DEVI void advance(RingPos& r, int ns) {
  if (++r.slot == ns) { r.slot = 0; r.parity ^= 1u; }
}

DEVI void advance(ProducerPos& r, int ns) {
  ++r.count;
  advance(static_cast<RingPos&>(r), ns);
}

// Whole tiles are dealt to the CTAs as evenly as they go: a GEMV phase of the step is a handful of tile-units per
// warp, so one tile more or less on a CTA moves the phase by a tenth of a microsecond, and no row of padding is
// ever streamed.
DEVI Slice slice_of(int rows, int paired, int cta, int ncta) {
  const int tiles = paired ? (rows + 7) >> 3 : (rows + 15) >> 4;
  const int base = tiles / ncta, rem = tiles % ncta;
  Slice s;
  s.t0 = cta * base + min(cta, rem);
  s.nt = base + (cta < rem ? 1 : 0);
  return s;
}

// Producer: issue every stage of one matrix slice, one copy each (a bulk copy costs ~0.2 us to issue whatever its
// size, so several small copies per stage would make the producer the bottleneck).
DEVI void produce(const Cta& c, const uint8_t* base, int nunit, const Slice& s, ProducerPos& rp, int lane) {
  const int NU = s.nt * nunit;
  const uint8_t* src = base + (size_t)s.t0 * nunit * kTileUnitBytes;
#pragma unroll 1
  for (int i0 = 0; i0 < NU; i0 += s.ups, advance(rp, c.p->ns)) {
    const int slot = rp.slot;
    if (!wait_bar(c, c.empty(slot), rp.parity, ERR_EMPTY, 200)) return;
    if (lane == 0) {
      const uint32_t bytes = (uint32_t)(min(s.ups, NU - i0) * kTileUnitBytes);
      mbar_expect_tx(c.full(slot), bytes);
      bulk_g2s(c.stage(slot), src + (size_t)i0 * kTileUnitBytes, bytes, c.full(slot));
    }
  }
}

// Cached tokens per attention ring stage: K rows in the first half of the stage, V rows in the second.
DEVI int kv_tokens_per_stage(const StepParams& p) {
  int t = min(kMaxKvTokens / (p.D / 64), p.stage_w / (4 * p.D));   // head_dim 128: 64, a team of two warps takes a block
  return t & ~((1 << p.log2P) - 1);
}

// Producer: the cached K/V rows [t0, t1) of one kv head, page by page (t0 is a multiple of the page size). Whole pages are
// copied; rows at or beyond t1 in the last page are ignored by the consumer.
DEVI void produce_kv(const Cta& c, const StepParams& p, const StepLayer& ly, int kvh, int t0, int t1, ProducerPos& rp, int lane) {
  const int tps = kv_tokens_per_stage(p);
  const uint32_t page_bytes = (uint32_t)(p.D * 2) << p.log2P;
#pragma unroll 1
  for (int t = t0; t < t1; t += tps, advance(rp, c.p->ns)) {
    const int slot = rp.slot;
    if (!wait_bar(c, c.empty(slot), rp.parity, ERR_EMPTY, 200)) return;
    const int pg0 = t >> p.log2P, npg = (min(tps, t1 - t) + (1 << p.log2P) - 1) >> p.log2P;
    uint8_t* dst = c.stage(slot);
    if (lane == 0) mbar_expect_tx(c.full(slot), 2 * npg * page_bytes);
    __syncwarp();
#pragma unroll 1
    for (int pg = lane; pg < npg; pg += 32) {
      const size_t off = ((size_t)p.bt[pg0 + pg] * p.n_kv + kvh) * page_bytes;
      bulk_g2s(dst + pg * page_bytes, reinterpret_cast<const uint8_t*>(ly.kc) + off, page_bytes, c.full(slot));
      bulk_g2s(dst + (size_t)tps * p.D * 2 + pg * page_bytes, reinterpret_cast<const uint8_t*>(ly.vc) + off,
               page_bytes, c.full(slot));
    }
  }
}

// One tile-unit block (at byte `tu` of shared memory: 32-bit offsets from one base, not pointers, which would take 64-bit arithmetic for
// every block) against unit u of x: the dot products of row slots g (ya) and g + 8 (yb)
// over the unit's 128 columns, scaled and with the zero-point term; meaningful on lanes t == 0.
// Lane (g, t) reads 16 bytes of row slot g and of row slot g + 8 (columns 32 t .. 32 t + 31 of the unit); lanes
// (0, t) carry the hi digits of the matching 32 activations as the B operand, lanes (1, t) the lo digits, the other
// lanes zeros. Four MMAs in two independent chains.
DEVI void tile_unit(const Cta& c, uint32_t tu, int u, int lane, float& ya, float& yb) {
  const int g = lane >> 2, t = lane & 3;
  uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
  if (g < 2) {
    const uint4* xp = reinterpret_cast<const uint4*>(step_smem + (uint32_t)(c.p->off_xin + 256 * u + 32 * (g * 4 + t)));
    x0 = xp[0];   // MMAs 0, 1: registers (m0 r0, m0 r1, m1 r0, m1 r1)
    x1 = xp[1];   // MMAs 2, 3
  }
  const uint4 wa = *reinterpret_cast<const uint4*>(step_smem + (tu + 16 * lane));
  const uint4 wb = *reinterpret_cast<const uint4*>(step_smem + (tu + 16 * lane) + 512);
  constexpr uint32_t kNib = 0x0F0F0F0Fu;
  int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
  mma16832_u8s8(c0, wa.x & kNib, wb.x & kNib, wa.y & kNib, wb.y & kNib, x0.x, x0.y);
  mma16832_u8s8(c1, (wa.x >> 4) & kNib, (wb.x >> 4) & kNib, (wa.y >> 4) & kNib, (wb.y >> 4) & kNib, x0.z, x0.w);
  mma16832_u8s8(c0, wa.z & kNib, wb.z & kNib, wa.w & kNib, wb.w & kNib, x1.x, x1.y);
  mma16832_u8s8(c1, (wa.z >> 4) & kNib, (wb.z >> 4) & kNib, (wa.w >> 4) & kNib, (wb.w >> 4) & kNib, x1.z, x1.w);
  // lanes t == 0: C columns 0 (hi digits) and 1 (lo digits) of rows g (c[0], c[1]) and g + 8 (c[2], c[3])
  const uint8_t* sz = step_smem + (tu + 4 * g) + 1024;
  const float2 sa = __half22float2(*reinterpret_cast<const half2*>(sz)), sc = __half22float2(*reinterpret_cast<const half2*>(sz + 32));
  const float2 xf = *reinterpret_cast<const float2*>(step_smem + (uint32_t)(c.p->off_xsum + 8 * u));
  const float xs = xf.x, resc = xf.y;
  const float va = (float)(((c0[0] + c1[0]) << 8) + (c0[1] + c1[1]));
  const float vb = (float)(((c0[2] + c1[2]) << 8) + (c0[3] + c1[3]));
  ya = fmaf(sa.x, fmaf(va, resc, -sa.y * xs), ya);
  yb = fmaf(sc.x, fmaf(vb, resc, -sc.y * xs), yb);
}

// The same for two blocks, of two tiles, against one unit of x: two independent chains.
DEVI void tile_unit2(const Cta& c, uint32_t tu, uint32_t tv, int u, int lane, float& ya, float& yb, float& za, float& zb) {
  tile_unit(c, tu, u, lane, ya, yb);
  tile_unit(c, tv, u, lane, za, zb);
}

// Consumer side of one matrix slice, one warp's share. The slice is the sequence of tile-unit blocks
// (tile 0 unit 0, tile 0 unit 1, ..., tile 1 unit 0, ...), `ups` of them per ring stage; warp w takes the blocks of
// units w, w + kNCW, ... of every tile, two at a time where the ring stage holds both (two independent instruction
// streams for the scheduler to interleave). Rows of 2048 weights are 16 units for 11 warps: sharing the last five between two warps
// each (half of a block's MMAs) evens the warps out on paper, and measured 20 us a token slower than leaving them. The activations are re-read from shared memory for every block: keeping
// them in registers across tiles was measured and loses - it pushes the kernel over its registers, and a spilled
// register costs an L2 round trip here. When the warp has passed its last unit of a tile, lanes t == 0 leave the
// two partial sums of rows g and g + 8 in part[warp][16 * tile + row slot]. A warp whose units do not exist
// (K < 1408) only keeps the ring's barriers moving.
//
// TILES: slices of whole tiles (Slice) have a loop of their own, which knows where a warp's one or two units of every tile are and takes
// two tiles at a time: a tile of 16 units on 11 warps takes 690 cycles in the general loop, which keeps track of tile, unit and stage,
// and 555 in a plain one over tiles (measured by themselves); with two tiles every warp has two chains in flight, also those with one
// unit of a tile. TinyLlama shape, us a token, this loop, 32-bit offsets instead of pointers into the ring, and the stages of 22: context 128
// 354 -> 339, 256 368 -> 353, 2048 400 -> 385, 8192 440 -> 423. Not in the STAGED form at head_dim 128, whose registers it exceeds (152 -> 157
// us for 4 layers, 32 kv heads). Two tiles at once in the general loop lost 3 %; four units of a row of 5632 at once, both stages, 1 %.
template <bool TILES>
DEVI void gemv(const Cta& c, const Mat& m, const Slice& s, float* part, int pstride, RingPos& rp, int warp, int lane,
               int trace_at) {
  const int g = lane >> 2, t = lane & 3;
  const int nunit = m.K >> 7, NU = s.nt * nunit;
  const bool active = warp < nunit;
  long long waited = 0;   // for the ring stages of the matrix
  if (TILES && s.whole) {
    const bool two = warp + kNCW < nunit;
    float* to = part + warp * pstride + g;
#pragma unroll 1
    for (int left = s.nt; left > 0; left -= s.whole, advance(rp, c.p->ns)) {
      const int slot = rp.slot;
      if (wait_full(c, slot, rp.parity, waited) && active) {
        uint32_t tu = (uint32_t)(c.p->off_ring + slot * c.p->stage_bytes + warp * kTileUnitBytes);
#pragma unroll 1
        for (int n = min(s.whole, left); n > 0;) {
          if (n > 1) {
            const uint32_t tv = tu + nunit * kTileUnitBytes;
            float ya = 0.f, yb = 0.f, za = 0.f, zb = 0.f;
            tile_unit2(c, tu, tv, warp, lane, ya, yb, za, zb);
            if (two) tile_unit2(c, tu + kNCW * kTileUnitBytes, tv + kNCW * kTileUnitBytes, warp + kNCW, lane, ya, yb, za, zb);
            if (t == 0) to[0] = ya, to[8] = yb, to[16] = za, to[24] = zb;
            n -= 2, tu += 2 * nunit * kTileUnitBytes, to += 32;
            continue;
          }
          float ya = 0.f, yb = 0.f, ya2 = 0.f, yb2 = 0.f;
          tile_unit(c, tu, warp, lane, ya, yb);
          if (two) tile_unit(c, tu + kNCW * kTileUnitBytes, warp + kNCW, lane, ya2, yb2);
          if (t == 0) to[0] = ya + ya2, to[8] = yb + yb2;
          --n, tu += nunit * kTileUnitBytes, to += 16;
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(c.empty(slot));
    }
    stamp_value(c, trace_at, waited);
    return;
  }
  int tl = 0, u = warp, idx = warp;   // the warp's next block: local tile, unit, place in the sequence
  float ya = 0.f, yb = 0.f;
#pragma unroll 1
  for (int i0 = 0; i0 < NU; i0 += s.ups, advance(rp, c.p->ns)) {
    const int slot = rp.slot;
    const bool ok = wait_full(c, slot, rp.parity, waited);
    const int end = min(NU, i0 + s.ups);
    const uint32_t sb = (uint32_t)(c.p->off_ring + slot * c.p->stage_bytes - i0 * kTileUnitBytes);   // block idx of the sequence is at sb + idx * 1088
    if (ok && active) {
#pragma unroll 1
      while (idx < end) {
        const bool two = u + kNCW < nunit && idx + kNCW < end;   // the next unit of the same tile is in this stage too
        float ya2 = 0.f, yb2 = 0.f;
        tile_unit(c, sb + (uint32_t)(idx * kTileUnitBytes), u, lane, ya, yb);
        if (two) tile_unit(c, sb + (uint32_t)((idx + kNCW) * kTileUnitBytes), u + kNCW, lane, ya2, yb2);
        ya += ya2;
        yb += yb2;
        const int step = two ? 2 * kNCW : kNCW;
        u += step;
        if (u >= nunit) {
          if (t == 0) {
            part[warp * pstride + 16 * tl + g] = ya;
            part[warp * pstride + 16 * tl + g + 8] = yb;
          }
          ya = yb = 0.f;
          ++tl;
          u = warp;
          idx = tl * nunit + warp;
        } else {
          idx += step;
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(c.empty(slot));
  }
  stamp_value(c, trace_at, waited);
}

// Sum of one row slot over the nwa warps that hold a share of it, always in the same order: pairs, then the pair sums. The
// loads are issued together; a loop would make every one wait for the add before it.
DEVI float sum_partials(const float* p, int pstride, int nwa) {
  float v[kNCW];
#pragma unroll
  for (int k = 0; k < kNCW; ++k) v[k] = k < nwa ? p[k * pstride] : 0.f;
#pragma unroll
  for (int k = 0; k + 1 < kNCW; k += 2) v[k] += v[k + 1];
  float y = v[0];
#pragma unroll
  for (int k = 2; k < kNCW; k += 2) y += v[k];
  return y;
}

// After the barrier that follows gemv(): thread i adds the warps' partial sums of row slot i in a fixed order
// (deterministic), multiplies by f (the norm's factor, or 1) and emits the output: E[row] <- tagged y; gate|up: E[i] <- tagged half(silu(gate_i)) * up_i.
DEVI void reduce_emit(const Cta& c, const Mat& m, const Slice& s, const float* part, int pstride, uint32_t* E, float f, int tid) {
  const int nwa = min(kNCW, m.K >> 7);
  if (m.paired) {
#pragma unroll 1
    for (int i = tid; i < 8 * s.nt; i += kNT) {
      const int slot = 16 * (i >> 3) + (i & 7), o = 8 * s.t0 + i;
      if (o >= m.N) continue;
      const float ga = sum_partials(part + slot, pstride, nwa), up = sum_partials(part + slot + 8, pstride, nwa);
      const half h0 = __float2half(ga * f), h1 = __float2half(up * f);
      const float gf = __half2float(h0);
      const half sl = __float2half(__fdividef(gf, 1.f + __expf(-gf)));
      st_tagged(E + o, c.tagw | (uint32_t)__half_as_ushort(__hmul(sl, h1)));
    }
    return;
  }
#pragma unroll 1
  for (int i = tid; i < 16 * s.nt; i += kNT) {
    const int row = 16 * s.t0 + i;
    if (row < m.N) st_tagged(E + row, c.tagw | (uint32_t)__half_as_ushort(__float2half(sum_partials(part + i, pstride, nwa) * f)));
  }
}

// The same for the LM head: logits[row] <- y; returns the largest key of this thread's rows (argmax_key; 0 = none comparable).
DEVI unsigned long long emit_logits(const Cta& c, const Slice& s, int tid) {
  const StepParams& p = *c.p;
  unsigned long long best = 0ull;
  const int nwa = min(kNCW, p.H >> 7);
  const float f = norm_factor(c, p.H, p.eps);
#pragma unroll 1
  for (int i = tid; i < 16 * s.nt; i += kNT) {
    const int row = 16 * s.t0 + i;
    if (row >= p.V) continue;
    const half h = __float2half(sum_partials(c.part() + i, p.part_stride_head, nwa) * f);
    p.logits[row] = h;
    if (!__hisnan(h)) { const unsigned long long key = argmax_key(h, row); best = key > best ? key : best; }
  }
  return best;
}

// ---- attention -------------------------------------------------------------------------------------------------------
// The cut of a context of `pos` cached tokens: short ones by attention_head, longer ones in slices. With the wide exchange by
// attention_group: every CTA takes part and a CTA per head merges the slices in one more exchange (~1.3 us). Without it (STAGED) a
// layer's block has room for att_slices partials per query head: attention_head takes a slice of whole ring stages, and the CTAs
// that stage the attention output merge. (4 layers behind 8192 tokens, us a token: 32 kv heads x 128 559 with one CTA per head, 298 with
// four slices in the wide exchange, 268 this way. 32 / 4 heads x 64 without the wide exchange 152 with the groups of
// attention_group, kv heads x 4 CTAs, and 130 this way.) Build-time knobs for measurements: tokens per slice and where the sliced
// forms begin (the wide one by the bytes a CTA copies for one head).
#ifndef B200_STEP_SLICE_TOKENS
#define B200_STEP_SLICE_TOKENS 128
#endif
#ifndef B200_STEP_TWO_MIN
#define B200_STEP_TWO_MIN 512
#endif
#ifndef B200_STEP_STAGED_MIN
#define B200_STEP_STAGED_MIN 1152
#endif
template <bool STAGED>
DEVI AttPlan att_plan(const StepParams& p, int pos, uint32_t epoch) {
  AttPlan r;
  r.two = !STAGED && p.att_max > 1 && pos * p.D >= 64 * B200_STEP_TWO_MIN;
  r.staged = STAGED && pos >= B200_STEP_STAGED_MIN;
  const int want = (pos + B200_STEP_SLICE_TOKENS - 1) / B200_STEP_SLICE_TOKENS;
  const int A = r.two ? min(p.att_max, want) : (r.staged ? p.att_slices : 1);
  const int align = r.staged ? kv_tokens_per_stage(p) : max(16, 1 << p.log2P);
  r.per = max(align, ((pos + A - 1) / A + align - 1) / align * align);
  r.A = max(1, (pos + r.per - 1) / r.per);   // no slice is empty
  r.refresh = (epoch & 1023u) == 0;
  r.pos = pos;
  r.units = r.two ? p.att_groups * r.A : p.n_q * r.A;
  return r;
}

// Attention unit u of a layer: heads [h0, h0 + nh) of one kv head, context slice j.
struct AttUnit { int kvh, h0, nh, j; };
DEVI AttUnit att_unit(const StepParams& p, int u) {
  const int hpg = p.n_q / p.n_kv, nsub = (hpg + 7) >> 3, grp = u % p.att_groups, sub = grp % nsub;
  AttUnit r;
  r.kvh = grp / nsub;
  r.h0 = r.kvh * hpg + 8 * sub;
  r.nh = min(8, hpg - 8 * sub);
  r.j = u / p.att_groups;
  return r;
}

// Where slice j's partials go: the layer's block of the exchange (merged while staging) or of the wide exchange (two).
struct AttOut { uint32_t* o; uint32_t* lse; int lsew; };
DEVI AttOut att_out(const StepParams& p, int layer, bool two) {
  const int n_att = p.n_q * p.D;
  AttOut r;
  r.o = two ? p.att_xchg + (size_t)layer * p.att_layer_words
            : p.xchg + (size_t)layer * p.layer_words + (p.n_q + 2 * p.n_kv) * p.D;
  r.lse = r.o + (size_t)(two ? p.att_max : p.att_slices) * n_att;
  r.lsew = step_lse_words(two ? p.att_max : p.att_slices);
  return r;
}

// fp32 value as an fp16 value and the fp16 remainder, tagged
DEVI void st_lse(const Cta& c, uint32_t* p, float v) {
  const half hi = __float2half(v), lo = __float2half(v - __half2float(hi));
  st_tagged2(p, c.tagw | (uint32_t)__half_as_ushort(hi), c.tagw | (uint32_t)__half_as_ushort(lo));
}

// Every 1024th step: the partial slots this step leaves alone get the current tag (see "tagged exchange words"). CTA h + k ncta
// does head h.
__device__ __noinline__ void refresh_partials(const Cta c, int layer) {
  const StepParams& p = *c.p;
  const AttPlan pl = c.plan();
  const int tid = threadIdx.x, n_att = p.n_q * p.D;
  for (int h = blockIdx.x; h < p.n_q; h += gridDim.x) {
    for (int two = 0; two < 2; ++two) {
      const AttOut out = att_out(p, layer, two);
      const bool partials = two ? pl.two : pl.staged;   // this step writes A of them here; otherwise the layer's block has one output
      const int slots = two ? p.att_max : p.att_slices, used = partials ? pl.A : (two ? 0 : 1), used_l = partials ? pl.A + (pl.A & 1) : 0;
      for (int i = used * p.D + tid; i < slots * p.D; i += kNT) st_tagged(out.o + (size_t)(i / p.D) * n_att + h * p.D + i % p.D, c.tagw);
      for (int i = 2 * used_l + tid; slots > 0 && i < out.lsew; i += kNT) st_tagged(out.lse + (size_t)h * out.lsew + i, c.tagw);
    }
  }
}

// x <- the attention output, merged from the A slices of every head while it is staged: x = sum_j 2^(l_j - max l) o_j /
// sum_j 2^(l_j - max l). Lane l of the warp that owns unit u holds 4 values of one head. Not inlined: the one loop body that
// serves every phase of the step would have to find registers for it.
__device__ __noinline__ void stage_attn(const Cta c, int layer, int warp, int lane) {
  constexpr int NL = (kStepMaxAttSlices + 1) / 2;   // granules of log-sum-exp words per head
  const StepParams& p = *c.p;
  const AttOut in = att_out(p, layer, false);
  const int nunit = p.n_att >> 7, A = c.plan().A;
  const uint32_t lbase = (uint32_t)(in.lse - in.o);
#pragma unroll 1
  for (int u = warp; u < nunit; u += kNCW) {
    const int i = 128 * u + 4 * lane, h = i / p.D;
    // While the slices are still at work the warp polls the log-sum-exp words only: one or two addresses per head, the same for all
    // lanes of a head, instead of A granules per lane - every CTA polls. When those are there the outputs are too, or nearly (the
    // second poll checks their tags all the same).
    uint32_t loff[NL], ooff[kStepMaxAttSlices];
#pragma unroll
    for (int g = 0; g < NL; ++g) loff[g] = lbase + (uint32_t)(h * in.lsew + 4 * g);
#pragma unroll
    for (int k = 0; k < kStepMaxAttSlices; ++k) ooff[k] = (uint32_t)(k * p.n_att + i);
    uint2 lv[NL], v[kStepMaxAttSlices];
    poll_list(c, in.o, loff, (1u << ((A + 1) >> 1)) - 1u, lv);
    poll_list(c, in.o, ooff, (1u << A) - 1u, v);
    float lse[kStepMaxAttSlices], M = -CUDART_INF_F;
#pragma unroll
    for (int k = 0; k < kStepMaxAttSlices; ++k) {
      lse[k] = -CUDART_INF_F;
      if (k < A) {
        const float2 f = __half22float2(as_h2((k & 1) ? lv[k >> 1].y : lv[k >> 1].x));   // (value, remainder)
        lse[k] = f.x + f.y;
        M = fmaxf(M, lse[k]);
      }
    }
    float W = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < kStepMaxAttSlices; ++k) {
      if (k < A) {
        const float w = exp2f(lse[k] - M);   // M is finite: no slice is empty
        const float2 x01 = __half22float2(as_h2(v[k].x)), x23 = __half22float2(as_h2(v[k].y));
        W += w;
        o[0] = fmaf(w, x01.x, o[0]), o[1] = fmaf(w, x01.y, o[1]), o[2] = fmaf(w, x23.x, o[2]), o[3] = fmaf(w, x23.y, o[3]);
      }
    }
    const float r = 1.f / W;
    put_unit(c, u, make_float4(o[0] * r, o[1] * r, o[2] * r, o[3] * r), lane);
  }
  __syncwarp();
}

DEVI uint4 lds16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// ---- short contexts: one CTA per query head -------------------------------------------------------------------------
// All consumer threads of the CTA, for unit u = head u % n_q (and, STAGED, context slice u / n_q; the last one takes the token of this
// step). q, k, v of this step come from the tagged qkv exchange, the cached tokens from ring stages filled by produce_kv. Lane
// (t = lane >> 3, c = lane & 7) of warp w owns token slot 4 w + t of a stage and dims [c D/8, (c+1) D/8) of it, on the fp32 pipes;
// each warp keeps a private online-softmax state, merged once at the end. Against attention_group: eight times the copies, but
// a head per CTA is less work on the way from q to the output, and up to a few hundred tokens that way is what counts (TinyLlama
// shape, context 128: 359 us a token, 376 with the groups).
template <int D, bool STAGED>
DEVI void attention_head(const Cta& c, const StepParams& p, const StepLayer& ly, uint32_t* E, int u, RingPos& rp, int tid,
                         int trace_at) {
  constexpr int D2 = D / 2, G4 = D / 4, DPL = D / 8;
  const int warp = tid >> 5, lane = tid & 31, ts = lane >> 3, ch = lane & 7, pos = c.plan().pos;
  const int h = STAGED ? u % p.n_q : u, hpg = p.n_q / p.n_kv, kvh = h / hpg;
  const int tps = kv_tokens_per_stage(p);
  const int t0 = STAGED ? u / p.n_q * c.plan().per : 0, len = STAGED ? min(c.plan().per, pos - t0) : pos;   // the slice's cached tokens
  const bool takes_new = !STAGED || t0 + len == pos;
  const int nst = (len + tps - 1) / tps;
  float* qf = reinterpret_cast<float*>(c.att());              // [D] rotated q * 1/sqrt(D)
  half* knew = reinterpret_cast<half*>(qf + D);           // [D] rotated k of this step
  half* vnew = knew + D;                                     // [D]
  half* raw = vnew + D;                                      // [3 D] un-rotated q, k, v
  float* wo = qf + 4 * D;                                 // [kNCW][D] per-warp outputs
  float* wm = wo + kNCW * D;                                 // [kNCW] per-warp max
  float* wl = wm + kNCW;                                     // [kNCW] per-warp sum
  const float* rope = c.rope();
  const int pmask = (1 << p.log2P) - 1;

  if (tid < 3 * G4) {
    const int which = tid / G4, g = tid % G4;
    const int head = which == 0 ? h : (which == 1 ? p.n_q + kvh : p.n_q + p.n_kv + kvh);
    reinterpret_cast<uint2*>(raw)[tid] = poll4(c, E + (size_t)head * D + 4 * g);
  }
  consumer_sync();
  if (tid < 2 * D) {
    const int slot_new = pos & pmask;
    const int page_new = reinterpret_cast<const int*>(rope)[D];
    const float cs = rope[tid % D2], sn = rope[D2 + tid % D2];
    const size_t row_new = ((((size_t)page_new * p.n_kv + kvh) << p.log2P) + slot_new) * D;
    if (tid < D) {
      const int i = tid % D2;
      const half* src = raw + (tid < D2 ? 0 : D);           // threads [0, D2): q pair i; [D2, D): k pair i
      const float a = __half2float(src[i]), b = __half2float(src[i + D2]);
      const half ra = __float2half(a * cs - b * sn), rb = __float2half(b * cs + a * sn);
      if (tid < D2) {
        const float scale = rsqrtf((float)D);
        qf[i] = __half2float(ra) * scale;
        qf[i + D2] = __half2float(rb) * scale;
      } else {
        knew[i] = ra;
        knew[i + D2] = rb;
        if (takes_new && h % hpg == 0) { ly.kc[row_new + i] = ra; ly.kc[row_new + i + D2] = rb; }
      }
    } else {
      const int i = tid - D;
      const half v = raw[2 * D + i];
      vnew[i] = v;
      if (takes_new && h % hpg == 0) ly.vc[row_new + i] = v;
    }
  }
  consumer_sync();

  stamp(c, trace_at);
  float qreg[DPL];
#pragma unroll
  for (int d = 0; d < DPL; ++d) qreg[d] = qf[ch * DPL + d];
  float m = -CUDART_INF_F, l = 0.f, acc[DPL];
#pragma unroll
  for (int d = 0; d < DPL; ++d) acc[d] = 0.f;

  // Fold kKvRounds rounds of 4 tokens per warp into the warp's online-softmax state. Round r, token slot ts: the K row
  // at byte koff[r] of shared memory, the V row at voff[r], counted if valid[r] (a slot that is not valid reads this
  // step's own k, v - real data, masked by its score; stale bytes of the ring could be NaN patterns, and 0 * NaN
  // would poison the sum). The scores of all rounds are computed independently and share ONE max / rescale step, so
  // a ring stage costs one dependent chain (loads, dot product, shuffles, exponentials, accumulate) whatever its
  // token count; the round count is fixed so that the chain carries no predicates.
  auto fold = [&](const uint32_t (&koff)[kKvRounds], const uint32_t (&voff)[kKvRounds], const bool (&valid)[kKvRounds]) {
    float s[kKvRounds];
#pragma unroll
    for (int r = 0; r < kKvRounds; ++r) {
      const half* kp = reinterpret_cast<const half*>(step_smem + koff[r]);
      float kf[DPL], a0 = 0.f, a1 = 0.f;
#pragma unroll
      for (int d8 = 0; d8 < DPL; d8 += 8) unpack8(*reinterpret_cast<const uint4*>(kp + d8), kf + d8);
#pragma unroll
      for (int d = 0; d < DPL; d += 2) { a0 = fmaf(kf[d], qreg[d], a0); a1 = fmaf(kf[d + 1], qreg[d + 1], a1); }
      float a = a0 + a1;
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      a += __shfl_xor_sync(0xffffffffu, a, 2);
      a += __shfl_xor_sync(0xffffffffu, a, 4);
      s[r] = valid[r] ? a : -CUDART_INF_F;
    }
    float mw = s[0];
#pragma unroll
    for (int r = 1; r < kKvRounds; ++r) mw = fmaxf(mw, s[r]);
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 8));
    mw = fmaxf(mw, __shfl_xor_sync(0xffffffffu, mw, 16));
    const float mn = fmaxf(m, mw);
    if (mn == -CUDART_INF_F) return;           // nothing valid yet in this warp (warp-uniform)
    const float alpha = __expf(m - mn);
    m = mn;
    l *= alpha;
#pragma unroll
    for (int d = 0; d < DPL; ++d) acc[d] *= alpha;
#pragma unroll
    for (int r = 0; r < kKvRounds; ++r) {
      const half* vp = reinterpret_cast<const half*>(step_smem + voff[r]);
      const float pr = __expf(s[r] - mn);      // a masked slot: e^(-inf) = 0
      l += pr;
      float vf[DPL];
#pragma unroll
      for (int d8 = 0; d8 < DPL; d8 += 8) unpack8(*reinterpret_cast<const uint4*>(vp + d8), vf + d8);
#pragma unroll
      for (int d = 0; d < DPL; ++d) acc[d] = fmaf(pr, vf[d], acc[d]);
    }
  };

  // The cached tokens come stage by stage from the ring. The token of this step (rotated k, v in the attention scratch)
  // rides along as token number nt of the (last slice's) last stage: a stage holds at most kMaxKvTokens tokens and the warps' slots cover
  // 4 kNCW kKvRounds > kMaxKvTokens, so there is always a slot for it and it costs no chain of its own.
  static_assert(4 * kNCW * kKvRounds > kMaxKvTokens, "a stage needs a spare slot for the token of this step");
  const uint32_t knew_off = (uint32_t)(reinterpret_cast<const uint8_t*>(knew) - step_smem) + ch * DPL * 2;
  const uint32_t vnew_off = (uint32_t)(reinterpret_cast<const uint8_t*>(vnew) - step_smem) + ch * DPL * 2;
  long long waited = 0;
#pragma unroll 1
  for (int st = 0; st < nst || (nst == 0 && st == 0); ++st) {   // an empty cache: one pass without a ring stage
    const bool have = st < nst, last = st + 1 >= nst;
    const int slot = rp.slot;
    const bool ok = have ? wait_full(c, slot, rp.parity, waited) : true;
    const uint32_t kbase = c.p->off_ring + (uint32_t)slot * c.p->stage_bytes + ch * DPL * 2;
    const uint32_t vbase = kbase + (uint32_t)tps * D * 2;
    const int nt = have ? min(tps, len - st * tps) : 0;
    if (ok) {
      uint32_t koff[kKvRounds], voff[kKvRounds];
      bool valid[kKvRounds];
#pragma unroll
      for (int r = 0; r < kKvRounds; ++r) {
        const int jt = 4 * warp + ts + 4 * kNCW * r;   // token slot of the stage
        valid[r] = jt < nt || (takes_new && last && jt == nt);
        koff[r] = jt < nt ? kbase + (uint32_t)jt * (D * 2) : knew_off;
        voff[r] = jt < nt ? vbase + (uint32_t)jt * (D * 2) : vnew_off;
      }
      fold(koff, voff, valid);
    }
    if (have) {
      __syncwarp();
      if (lane == 0) mbar_arrive(c.empty(slot));
      advance(rp, c.p->ns);
    }
  }
  stamp(c, trace_at + 1);
  stamp_value(c, trace_at + 4, waited);   // a duration: what warp 0 waited for the K/V stages

  // merge: token slots inside the warp, then the warps
  float lw = l;
  lw += __shfl_xor_sync(0xffffffffu, lw, 8);
  lw += __shfl_xor_sync(0xffffffffu, lw, 16);
#pragma unroll
  for (int d = 0; d < DPL; ++d) {
    acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 8);
    acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], 16);
  }
  if (ts == 0) {
#pragma unroll
    for (int d = 0; d < DPL; ++d) wo[warp * D + ch * DPL + d] = acc[d];
    if (ch == 0) { wm[warp] = m; wl[warp] = lw; }
  }
  consumer_sync();
  if (tid < D) {
    float M = -CUDART_INF_F;
#pragma unroll
    for (int w = 0; w < kNCW; ++w) M = fmaxf(M, wm[w]);
    float o = 0.f, L = 0.f;
#pragma unroll
    for (int w = 0; w < kNCW; ++w) {
      const float a = __expf(wm[w] - M);   // a warp that saw no token: e^(-inf) = 0
      o = fmaf(a, wo[w * D + tid], o);
      L = fmaf(a, wl[w], L);
    }
    st_tagged(E + p.n_qkv + (size_t)u * D + tid, c.tagw | (uint32_t)__half_as_ushort(__float2half(o / L)));   // slot u / n_q, head h
    if (STAGED && c.plan().staged && tid == 0) {
      const int lsew = step_lse_words(p.att_slices), j = u / p.n_q;
      uint32_t* lp = E + p.n_qkv + (size_t)p.att_slices * p.n_att + (size_t)h * lsew + 2 * j;
      st_lse(c, lp, (M + __logf(L)) * 1.44269504088896340736f);
      if ((c.plan().A & 1) && takes_new) st_tagged2(lp + 2, c.tagw | 0xFC00u, c.tagw);   // the other half of the last granule: -inf
    }
  }
  stamp(c, trace_at + 2);
}

// Scratch of attention_group behind Cta::att().
template <int D>
struct AttScratch {
  half q[8][D + 8];              // rotated queries (padded rows)
  half k[D], v[D];               // rotated k and v of this step
  float m[kNCW][8], l[kNCW][8];  // per warp and head: running maximum (base-2 units) and sum
  float o[kNCW][8][65];          // per warp and head: un-normalised output, 64 dims
};

// All consumer threads of the CTA. q, k, v of this step come from the tagged qkv exchange, the slice's cached tokens from ring
// stages filled by produce_kv; the last slice also takes the token of this step and writes it to the cache. A block of 16
// tokens is one warp's work (block b of the slice: warp b mod kNCW), laid out as in paged_attn_mma_kernel: the heads are rows
// 0-7 of the MMAs; K and V fragments are read from the row-major pages by permuting the contraction index. The probabilities
// enter the second contraction twice, as fp16 value and as fp16 remainder, so they count with the precision of fp32.
template <int D>
DEVI RingPos attention_group(const Cta& c, int layer, int u, RingPos rp, int trace_at) {
  constexpr int HALVES = D / 64, TEAMS = kNCW / HALVES, CH = D / 32, NB = 8, D2 = D / 2, D4 = D / 4, PG = D / 8;
  const int tid = threadIdx.x;
  const StepParams& p = *c.p;
  const AttPlan& pl = c.plan();   // in shared memory, re-read where it is needed
  const AttUnit un = att_unit(p, u);
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  AttScratch<D>& sc = *reinterpret_cast<AttScratch<D>*>(c.att());
  const int t_begin = un.j * pl.per, t_end = min(pl.pos, t_begin + pl.per);
  const bool takes_new = un.j == pl.A - 1;

  // q of the group's heads (and k, v): a thread takes dims i .. i + 3 and their rotation partners i + D/2 ..
  if (tid < (un.nh + (takes_new ? 2 : 0)) * PG) {
    const int which = tid / PG, i = 4 * (tid % PG);
    const int row = which < un.nh ? un.h0 + which : (which == un.nh ? p.n_q : p.n_q + p.n_kv) + un.kvh;
    uint2 r[2];
    poll_many<2>(c, p.xchg + (size_t)layer * p.layer_words + (size_t)row * D + i, D2, 2, r);
    if (which <= un.nh) {
      const float4 cs = *reinterpret_cast<const float4*>(c.rope() + i), sn = *reinterpret_cast<const float4*>(c.rope() + D2 + i);
      const float2 a0 = __half22float2(as_h2(r[0].x)), a1 = __half22float2(as_h2(r[0].y));
      const float2 b0 = __half22float2(as_h2(r[1].x)), b1 = __half22float2(as_h2(r[1].y));
      r[0].x = as_u32(__floats2half2_rn(a0.x * cs.x - b0.x * sn.x, a0.y * cs.y - b0.y * sn.y));
      r[0].y = as_u32(__floats2half2_rn(a1.x * cs.z - b1.x * sn.z, a1.y * cs.w - b1.y * sn.w));
      r[1].x = as_u32(__floats2half2_rn(b0.x * cs.x + a0.x * sn.x, b0.y * cs.y + a0.y * sn.y));
      r[1].y = as_u32(__floats2half2_rn(b1.x * cs.z + a1.x * sn.z, b1.y * cs.w + a1.y * sn.w));
    }
    half* dst = which < un.nh ? sc.q[which] : (which == un.nh ? sc.k : sc.v);
    *reinterpret_cast<uint2*>(dst + i) = r[0];
    *reinterpret_cast<uint2*>(dst + D2 + i) = r[1];
    if (which >= un.nh && un.h0 == un.kvh * (p.n_q / p.n_kv)) {   // one unit of the kv head appends the row
      const int page = reinterpret_cast<const int*>(c.rope())[D], slot = pl.pos & ((1 << p.log2P) - 1);
      half* row_new = (which == un.nh ? c.layer(layer).kc : c.layer(layer).vc) + ((((size_t)page * p.n_kv + un.kvh) << p.log2P) + slot) * D;
      *reinterpret_cast<uint2*>(row_new + i) = r[0];
      *reinterpret_cast<uint2*>(row_new + D2 + i) = r[1];
    }
  }
  consumer_sync();
  stamp(c, trace_at);

  const float sl2 = 1.44269504088896340736f * rsqrtf((float)D);   // scores in base-2 units
  // head_dim 128: two warps share a block's scores and take 64 output dims each (32 accumulators more would spill)
  const int team = warp / HALVES, dim0 = 64 * (warp % HALVES);
  float m = -CUDART_INF_F, l = 0.f, acc[NB][2];
#pragma unroll
  for (int n = 0; n < NB; ++n) acc[n][0] = acc[n][1] = 0.f;

  const uint32_t qaddr = smem_u32(&sc.q[g][t * D4]), kaddr = smem_u32(sc.k), vaddr = smem_u32(sc.v);
  const int tps = kv_tokens_per_stage(p), bps = tps >> 4;   // tokens and blocks per stage
  int bid = 0, nblk = 0;                                     // first block of the stage mod kNCW; blocks of the slice
  long long waited = 0;
#pragma unroll 1
  for (int t0 = t_begin; t0 < t_end || nblk == 0; t0 += tps) {   // an empty cache: one pass without a ring stage
    const bool have = t0 < t_end, last = t0 + tps >= t_end;
    const int slot = rp.slot;
    const bool ok = have ? wait_full(c, slot, rp.parity, waited) : true;
    const int nt = have ? min(tps, t_end - t0) : 0, ntot = nt + (takes_new && last ? 1 : 0);   // the new token rides behind the last one
    const uint32_t kst = smem_u32(c.stage(slot)), vst = kst + (uint32_t)(tps * D * 2);
    int b = team - bid;
    if (b < 0) b += TEAMS;
    if (ok && 16 * b < ntot && team < TEAMS) {   // a stage holds at most TEAMS blocks (and one token): one per team
      const int tok0 = 16 * b;
      float s[2][2];
#pragma unroll
      for (int nb = 0; nb < 2; ++nb) s[nb][0] = s[nb][1] = 0.f;
      {
        // a row past the stage's tokens: this step's own (finite; masked unless it is its turn)
        const int j0 = tok0 + g, j1 = j0 + 8;
        const uint32_t k0 = (j0 < nt ? kst + j0 * (2 * D) : kaddr) + t * (2 * D4), k1 = (j1 < nt ? kst + j1 * (2 * D) : kaddr) + t * (2 * D4);
#pragma unroll
        for (int ch = 0; ch < CH; ++ch) {   // k-steps 2 ch and 2 ch + 1: dims t D/4 + 8 ch + {0 .. 3 | 4 .. 7}; row g = head g, zero beyond the group
          uint4 q4 = lds16(qaddr + 16 * ch);
          if (g >= un.nh) q4 = make_uint4(0u, 0u, 0u, 0u);
          const uint4 ka = lds16(k0 + 16 * ch), kb = lds16(k1 + 16 * ch);
          mma16816_top(s[0], q4.x, q4.y, ka.x, ka.y);
          mma16816_top(s[1], q4.x, q4.y, kb.x, kb.y);
          mma16816_top(s[0], q4.z, q4.w, ka.z, ka.w);
          mma16816_top(s[1], q4.z, q4.w, kb.z, kb.w);
        }
      }
      float pr[4];   // head g, tokens tok0 + 8 nb + 2 t + {0, 1}
#pragma unroll
      for (int nb = 0; nb < 2; ++nb)
#pragma unroll
        for (int e = 0; e < 2; ++e) pr[2 * nb + e] = tok0 + 8 * nb + 2 * t + e < ntot ? s[nb][e] * sl2 : -CUDART_INF_F;
      float mx = fmaxf(fmaxf(pr[0], pr[1]), fmaxf(pr[2], pr[3]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float mn = fmaxf(m, mx), alpha = exp2f(m - mn);   // finite: token tok0 counts
      m = mn;
#pragma unroll
      for (int e = 0; e < 4; ++e) pr[e] = exp2f(pr[e] - mn);
      l = fmaf(l, alpha, (pr[0] + pr[1]) + (pr[2] + pr[3]));
#pragma unroll
      for (int n = 0; n < NB; ++n) acc[n][0] *= alpha, acc[n][1] *= alpha;
      const half2 h01 = __floats2half2_rn(pr[0], pr[1]), h23 = __floats2half2_rn(pr[2], pr[3]);
      const float2 f01 = __half22float2(h01), f23 = __half22float2(h23);
      const uint32_t hi0 = as_u32(h01), hi2 = as_u32(h23);
      const uint32_t lo0 = as_u32(__floats2half2_rn(pr[0] - f01.x, pr[1] - f01.y)), lo2 = as_u32(__floats2half2_rn(pr[2] - f23.x, pr[3] - f23.y));
      uint32_t vr[4];   // V rows of tokens 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int jt = tok0 + 2 * t + (e & 1) + 8 * (e >> 1);
        vr[e] = (jt < nt ? vst + jt * (2 * D) : vaddr) + 16 * g + 2 * dim0;
      }
      {
        const uint4 v0 = lds16(vr[0]), v1 = lds16(vr[1]), v2 = lds16(vr[2]), v3 = lds16(vr[3]);
        const uint32_t w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
        const uint32_t w2[4] = {v2.x, v2.y, v2.z, v2.w}, w3[4] = {v3.x, v3.y, v3.z, v3.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t sel = e ? 0x7632u : 0x5410u, b0 = __byte_perm(w0[i], w1[i], sel), b1 = __byte_perm(w2[i], w3[i], sel);
            mma16816_top(acc[2 * i + e], hi0, hi2, b0, b1);
            mma16816_top(acc[2 * i + e], lo0, lo2, b0, b1);
          }
      }
    }
    nblk += (ntot + 15) >> 4;
    bid += bps;
    while (bid >= TEAMS) bid -= TEAMS;
    if (have) {
      __syncwarp();
      if (lane == 0) mbar_arrive(c.empty(slot));
      advance(rp, c.p->ns);
    }
  }
  stamp(c, trace_at + 1);
  stamp_value(c, trace_at + 4, waited);   // a duration: what warp 0 waited for the K/V stages

  // merge the teams: acc[n][e] = O[head g][dim0 + 8 (2 t + e) + n]
  const int nw = min(TEAMS, nblk);
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  if (team < nw) {
    if (t == 0) sc.m[warp][g] = m, sc.l[warp][g] = l;
#pragma unroll
    for (int n = 0; n < NB; ++n)
#pragma unroll
      for (int e = 0; e < 2; ++e) sc.o[warp][g][8 * (2 * t + e) + n] = acc[n][e];
  }
  consumer_sync();
  const AttOut out = att_out(p, layer, pl.two);
#pragma unroll 1
  for (int i = tid; i < un.nh * D2; i += kNT) {
    const int h = i / D2, d = 2 * (i % D2), w0 = d / 64;   // warps w0, w0 + HALVES, ... hold these dims
    float f[TEAMS], M = -CUDART_INF_F, L = 0.f, o0 = 0.f, o1 = 0.f;   // unrolled: the teams' loads are in flight together
#pragma unroll
    for (int k = 0; k < TEAMS; ++k) {
      f[k] = k < nw ? sc.m[k * HALVES][h] : -CUDART_INF_F;
      M = fmaxf(M, f[k]);
    }
#pragma unroll
    for (int k = 0; k < TEAMS; ++k) {
      if (k < nw) {
        const float w = exp2f(f[k] - M);
        o0 = fmaf(w, sc.o[k * HALVES + w0][h][d % 64], o0);
        o1 = fmaf(w, sc.o[k * HALVES + w0][h][d % 64 + 1], o1);
        L = fmaf(w, sc.l[k * HALVES][h], L);
      }
    }
    const float r = 1.f / L;
    st_tagged2(out.o + (size_t)un.j * (p.n_q * D) + (size_t)(un.h0 + h) * D + d, c.tagw | (uint32_t)__half_as_ushort(__float2half(o0 * r)),
               c.tagw | (uint32_t)__half_as_ushort(__float2half(o1 * r)));
    if (d == 0) {
      uint32_t* lp = out.lse + (size_t)(un.h0 + h) * out.lsew + 2 * un.j;
      st_lse(c, lp, M + __log2f(L));
      if ((pl.A & 1) && un.j == pl.A - 1) st_tagged2(lp + 2, c.tagw | 0xFC00u, c.tagw);   // the other half of the last granule: -inf
    }
  }
  stamp(c, trace_at + 2);
  return rp;   // the caller's barrier comes before the scratch is used again
}

// Two-level form: the attention output of head h from its A slices, by all consumer threads of one CTA. Thread (dims 4 k .. 4 k + 3,
// row s) folds slices s, s + rows, ...; the rows meet in shared memory.
template <int D>
DEVI void merge_head(const Cta& c, int layer, int h) {
  constexpr int G = D / 4, ROWS = kNT / G;
  const int tid = threadIdx.x;
  const StepParams& p = *c.p;
  const int A = c.plan().A, k = tid % G, row = tid / G, n_att = p.n_q * D;
  const AttOut in = att_out(p, layer, true);
  float* acc_s = reinterpret_cast<float*>(c.att());   // [ROWS][D]
  float* m_s = acc_s + ROWS * D;                      // [ROWS] maximum, [ROWS] weight
  float M = -CUDART_INF_F, W = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};
  if (row < ROWS) {
#pragma unroll 1
    for (int j = row; j < A; j += 2 * ROWS) {
      const int j2 = j + ROWS;
      const uint32_t mask = j2 < A ? 15u : 5u;
      uint32_t off[4];
      off[0] = (uint32_t)(j * n_att + h * D + 4 * k);
      off[1] = (uint32_t)(j2 * n_att + h * D + 4 * k);
      off[2] = (uint32_t)(in.lse - in.o) + (uint32_t)(h * in.lsew + 4 * (j >> 1));
      off[3] = (uint32_t)(in.lse - in.o) + (uint32_t)(h * in.lsew + 4 * (j2 >> 1));
      uint2 v[4];
      poll_list<4>(c, in.o, off, mask, v);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (e && j2 >= A) break;
        const float2 f = __half22float2(as_h2(((e ? j2 : j) & 1) ? v[2 + e].y : v[2 + e].x));
        const float2 x01 = __half22float2(as_h2(v[e].x)), x23 = __half22float2(as_h2(v[e].y));
        const float lse = f.x + f.y, Mn = fmaxf(M, lse), a = exp2f(M - Mn), w = exp2f(lse - Mn);
        W = fmaf(W, a, w);
        o[0] = fmaf(o[0], a, w * x01.x), o[1] = fmaf(o[1], a, w * x01.y);
        o[2] = fmaf(o[2], a, w * x23.x), o[3] = fmaf(o[3], a, w * x23.y);
        M = Mn;
      }
    }
    *reinterpret_cast<float4*>(acc_s + row * D + 4 * k) = make_float4(o[0], o[1], o[2], o[3]);
    if (k == 0) m_s[row] = M, m_s[ROWS + row] = W;
  }
  consumer_sync();
  if (tid < D) {
    float Mx = -CUDART_INF_F, Wt = 0.f, y = 0.f;
    const int rows = min(ROWS, A);
    for (int r = 0; r < rows; ++r) Mx = fmaxf(Mx, m_s[r]);
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
      const float f = exp2f(m_s[r] - Mx);
      Wt = fmaf(f, m_s[ROWS + r], Wt);
      y = fmaf(f, acc_s[r * D + tid], y);
    }
    st_tagged(att_out(p, layer, false).o + (size_t)h * D + tid, c.tagw | (uint32_t)__half_as_ushort(__float2half(y / Wt)));
  }
}

// The sliced form, all of a layer's work of this CTA. Not inlined: it would take registers from the loop that serves every phase of
// the step. False: the step is aborting.
struct AttDone { RingPos rp; bool ok; };
template <int D>
__device__ __noinline__ AttDone attention_sliced(const Cta c, int layer, RingPos rp, int trace_at) {
  const StepParams& p = *c.p;
#pragma unroll 1
  for (int u = blockIdx.x; u < c.plan().units; u += gridDim.x) {
    rp = attention_group<D>(c, layer, u, rp, trace_at);
    if (consumer_sync_or(*c.abort())) return AttDone{rp, false};
  }
  // the merging CTAs counted from the far end: they are the first to have no second unit
#pragma unroll 1
  for (int h = gridDim.x - 1 - blockIdx.x; h < p.n_q; h += gridDim.x) {
    merge_head<D>(c, layer, h);
    if (consumer_sync_or(*c.abort())) return AttDone{rp, false};
  }
  return AttDone{rp, true};
}

}  // namespace

// ---- the kernel ------------------------------------------------------------------------------------------------------
// STAGED: without the wide attention exchange (att_plan). A kernel of its own: the code that merges slices while staging, anywhere in
// the kernel, makes the loop that serves every phase spill 40 to 100 bytes.
template <int D, bool WIDE, bool STAGED>
__global__ void __launch_bounds__(kThreads, 1) decode_step_kernel(const __grid_constant__ StepParams p) {
  uint8_t* smem = step_smem;
  Cta c;
  c.p = &p;
  // the per-layer pointer table, copied once from global memory: every phase starts from these pointers, and a
  // global load in front of each would put an L2 round trip on the critical path ~10 times per layer
  StepLayer* lys = reinterpret_cast<StepLayer*>(smem + p.off_table);
  int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cta = blockIdx.x, ncta = gridDim.x;

  if (tid == 0) {
    for (int i = 0; i < p.ns; ++i) { mbar_init(c.full(i), 1); mbar_init(c.empty(i), kNCW); }
    *c.abort() = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // This CTA's tiles of the five matrix shapes of a step (qkv, o, gate|up, down, head): computed once (they involve
  // integer divisions) and kept in shared memory for producer and consumers.
  Slice* sl = reinterpret_cast<Slice*>(smem + 512);
  if (tid < 5) {
    const int rows = tid == 0 ? p.n_qkv : (tid == 2 ? p.I : (tid == 4 ? p.V : p.H));
    sl[tid] = slice_of(rows, tid == 2, cta, ncta);
    const int nunit = (tid == 1 ? p.n_att : tid == 3 ? p.I : p.H) >> 7;
    constexpr int kPass = 2 * kNCW;
    sl[tid].whole = nunit <= kPass && 2 * nunit <= p.ups ? p.ups / nunit : 0;
    sl[tid].ups = sl[tid].whole ? sl[tid].whole * nunit : sl[tid].nt == 1 && nunit > p.ups && nunit <= 2 * kPass ? min(kPass, p.ups) : p.ups;
  }
  {
    const uint4* src = reinterpret_cast<const uint4*>(p.layers);
    uint4* dst = reinterpret_cast<uint4*>(lys);
    for (int i = tid; i < p.L * (int)(sizeof(StepLayer) / 16); i += kThreads) dst[i] = __ldg(src + i);
  }
  const uint32_t epoch = ((volatile StepCtrl*)p.ctrl)->epoch + 1u;
  c.tagw = ((epoch % 65535u) + 1u) << 16;
  const int pos = p.pos[0];
  if (tid == 64) *reinterpret_cast<AttPlan*>(smem + 640) = att_plan<STAGED>(p, pos, epoch);
  __syncthreads();
  if (warp == kNCW) {
    // ================= producer =================
    ProducerPos rp;            // parity 1: the first pass over a fresh `empty` barrier does not wait
    rp.slot = 0, rp.parity = 1u, rp.count = 0;
    // one copy of the code for all matrices: it shares the instruction cache with the consumers
#pragma unroll 1
    for (int step = 0; step <= 4 * p.L && !*c.abort(); ++step) {
      const int l = step >> 2, k = step & 3;
      const bool head = l == p.L;
      const StepLayer& ly = lys[head ? 0 : l];
      produce(c, head ? (const uint8_t*)p.w_head : (const uint8_t*)ly.w[k], (k == 1 ? p.n_att : (k == 3 ? p.I : p.H)) >> 7,
              sl[head ? 4 : k], rp, lane);
      if (k == 0 && !head)
        for (int u = cta; u < c.plan().units && !*c.abort(); u += ncta) {
          const bool two = c.plan().two;
          const AttUnit un = att_unit(p, u);
          const int t0 = (two ? un.j : u / p.n_q) * c.plan().per;
          produce_kv(c, p, ly, two ? un.kvh : u % p.n_q / (p.n_q / p.n_kv), t0, min(c.plan().pos, t0 + c.plan().per), rp, lane);
        }
    }
    // Leave only when every copy issued has landed. On the normal path the consumers have waited on every full
    // barrier already; on abort, wait (bounded) for the full barriers of the stages still in the ring.
    if (*c.abort()) {
      const int it = rp.count;
      for (int k = max(0, it - c.p->ns); k < it; ++k) {
        const int slot = k % c.p->ns;
        for (int i = 0; i < kSpinLimit; ++i)
          if (mbar_try_wait(c.full(slot), (k / c.p->ns) & 1)) break;
      }
    }
    return;
  }

  // ================= consumers =================
#ifdef B200_STEP_TRACE
  // trace row of a CTA: kTraceHead slots (0 = start, 1 = keys exchanged, 2 = token written), then per layer
  // kTracePerLayer: per phase {staged, first weights there, GEMV done, barrier passed, emitted}, then attention
  // {q k v polled and rotated, cached tokens folded, warps merged and output stored, done, wait for K/V stages};
  // the LM head uses the slots of a layer L
  c.tr = p.trace ? p.trace + (size_t)cta * (kTraceHead + kTracePerLayer * (p.L + 1)) : nullptr;
#endif
  stamp(c, 0);
  RingPos rp = {0, 0u};
  // RoPE factors and the page of this step's token depend only on pos: the attention CTAs fetch them now, off the
  // critical path (first read behind the barriers of the first GEMV)
  if (cta < c.plan().units) {
    float* rope = c.rope();
    if (tid < (p.D >> 1)) {
      rope[tid] = p.cos_t[(size_t)pos * (p.D >> 1) + tid];
      rope[(p.D >> 1) + tid] = p.sin_t[(size_t)pos * (p.D >> 1) + tid];
    }
    if (tid == 0) reinterpret_cast<int*>(rope)[p.D] = p.bt[pos >> p.log2P];
  }
  // One loop body serves every GEMV of the step (4 per layer, then the LM head as "phase 0 of layer L"): the kernel
  // keeps a single copy of the staging, GEMV and attention code, which keeps the loop inside the instruction cache.
  const Mat head = {(const uint8_t*)p.w_head, p.V, p.H, 0};
#pragma unroll 1
  for (int step = 0; step <= 4 * p.L; ++step) {
    // Forget what is derived from these between phases: lane constants of the GEMV code would otherwise be kept in
    // registers through attention, and the kernel would spill.
    asm volatile("" : "+r"(tid), "+r"(warp), "+r"(lane));
    const int l = step >> 2, ph = step & 3;
    const bool is_head = l == p.L;
    const StepLayer& ly = lys[is_head ? 0 : l];
    uint32_t* E = p.xchg + (size_t)l * p.layer_words;
    uint32_t *Eqkv = E, *Eatt = E + p.n_qkv, *Else = Eatt + (size_t)p.att_slices * p.n_att;
    uint32_t *Eo = Else + p.n_q * step_lse_words(p.att_slices), *Eact = Eo + p.H, *Edown = Eact + p.I;
    Mat m;
    const uint32_t* Ein;
    const half* nw = nullptr;   // norm weight: non-null selects "residual add + RMSNorm" staging
    uint32_t* Eout;
    int n_in = p.H;
    if (ph == 0) {
      Ein = l == 0 ? nullptr : E - p.H;   // down of the previous layer: the last H words of its block
      nw = is_head ? p.norm_f : ly.ln1;
      m = is_head ? head : Mat{(const uint8_t*)ly.w[0], p.n_qkv, p.H, 0};
      Eout = Eqkv;
    } else if (ph == 1) {
      Ein = Eatt; n_in = p.n_att;
      m = Mat{(const uint8_t*)ly.w[1], p.H, p.n_att, 0};
      Eout = Eo;
    } else if (ph == 2) {
      Ein = Eo; nw = ly.ln2;
      m = Mat{(const uint8_t*)ly.w[2], p.I, p.H, 1};
      Eout = Eact;
    } else {
      Ein = Eact; n_in = p.I;
      m = Mat{(const uint8_t*)ly.w[3], p.H, p.I, 0};
      Eout = Edown;
    }
    const Slice s = sl[is_head ? 4 : ph];
    // the layers alternate between two partial-sum buffers (a slow thread may still add up phase n while a fast warp
    // writes phase n + 1); the head, last and largest, takes the whole area
    const int pstride = is_head ? p.part_stride_head : p.part_stride;
    float* part = c.part() + ((step & 1) && !is_head ? kNCW * p.part_stride : 0);
    if (nw) {
      const half* emb_row = nullptr;
      if (step == 0) {
        // A token id outside the embedding table (a caller's mistake) must not become an address: row 0 is read
        // instead and the step reports it.
        long long tok_in = p.tok[0];
        if (tok_in < 0 || tok_in >= p.V) {
          if (cta == 0 && tid == 0) atomicCAS(&p.ctrl->error, 0, ERR_TOKEN);
          tok_in = 0;
        }
        emb_row = p.emb + (size_t)tok_in * p.H;
      }
      stage_norm<WIDE ? kWideBatchNorm : kBatchNorm>(c, Ein, emb_row, nw, n_in, warp, lane);
    }
    else if (s.nt > 0) {
      if (STAGED && ph == 1 && c.plan().staged) stage_attn(c, l, warp, lane);
      else stage_plain<WIDE ? kWideBatch : kBatch>(c, Ein, n_in, warp, lane);
    }
    const int tr_at = kTraceHead + kTracePerLayer * l + kTracePerPhase * ph;
    stamp(c, tr_at);
    gemv<!(STAGED && D == 128)>(c, m, s, part, pstride, rp, warp, lane, tr_at + 1);
    stamp(c, tr_at + 2);
    if (consumer_sync_or(*c.abort())) return;
    stamp(c, tr_at + 3);
    if (is_head) break;
    reduce_emit(c, m, s, part, pstride, Eout, nw ? norm_factor(c, p.H, p.eps) : 1.f, tid);
    stamp(c, tr_at + 4);
    if (ph == 0) {
      if (c.plan().refresh) refresh_partials(c, l);
      const int tr_att = kTraceHead + kTracePerLayer * l + 4 * kTracePerPhase;
      if (!STAGED && c.plan().two) {
        const AttDone d = attention_sliced<D>(c, l, rp, tr_att);
        if (!d.ok) return;
        rp = d.rp;
      } else {
        for (int u = cta; u < (STAGED ? c.plan().units : p.n_q); u += ncta) {
          attention_head<D, STAGED>(c, p, ly, E, u, rp, tid, tr_att);
          if (consumer_sync_or(*c.abort())) return;
        }
      }
      stamp(c, kTraceHead + kTracePerLayer * l + 4 * kTracePerPhase + 3);
    }
  }
  // this CTA's candidate: max over its threads' keys
  unsigned long long best = emit_logits(c, sl[4], tid);
  stamp(c, kTraceHead + kTracePerLayer * p.L + 4);
  unsigned long long* keys = c.keys();
  {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
      best = other > best ? other : best;
    }
  }
  if (lane == 0) keys[warp] = best;
  if (consumer_sync_or(*c.abort())) return;
  stamp(c, 1);
  uint32_t* Earg = p.xchg + (size_t)p.L * p.layer_words;   // [ncta][4] words: idx low 16, idx high 16, value key, valid
  if (tid == 0) {
    unsigned long long b = 0ull;
    for (int k = 0; k < kNCW; ++k) b = keys[k] > b ? keys[k] : b;
    const uint32_t idx = 0x7FFFFFFFu - (uint32_t)(b & 0xFFFFFFFFu), val = (uint32_t)(b >> 32) & 0xFFFFu;
    uint32_t* e = Earg + 4 * cta;
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(e), "r"(c.tagw | (idx & 0xFFFFu)),
                 "r"(c.tagw | (idx >> 16)), "r"(c.tagw | val), "r"(c.tagw | (b ? 1u : 0u))
                 : "memory");
  }
  if (cta == 0) {
    unsigned long long b = 0ull;
    for (int k = tid; k < ncta; k += kNT) {
      const uint2 v = poll4(c, Earg + 4 * k);
      const uint32_t idx = v.x, val = v.y & 0xFFFFu, valid = v.y >> 16;
      if (valid) {
        const unsigned long long key = ((unsigned long long)val << 32) | (uint32_t)(0x7FFFFFFFu - idx);
        b = key > b ? key : b;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, b, o);
      b = other > b ? other : b;
    }
    if (lane == 0) keys[kNCW + warp] = b;
    consumer_sync();
    if (tid == 0 && !*c.abort()) {
      for (int k = 0; k < kNCW; ++k) b = keys[kNCW + k] > b ? keys[kNCW + k] : b;
      // b == 0: no logit was comparable (all NaN). torch.argmax, which the reference uses, answers with a valid
      // index in that case; token 0 is this kernel's answer.
      const long long t = b ? (long long)(0x7FFFFFFF - (int)(b & 0xFFFFFFFFu)) : 0ll;
      p.tok[0] = t;
      if (p.history) p.history[pos] = t;
      p.pos[0] = pos + 1;
      p.ctrl->epoch = epoch;
      stamp(c, 2);
    }
  }
}

// Lays the fixed areas out behind the header (sizes in, offsets out); returns where the ring starts. The attention scratch shares
// the activations' area where that is large enough: a GEMV's x is dead when attention runs and the other way round.
size_t decode_step_plan_smem(StepParams& p, int resid_bytes, int xin_bytes, int xsum_bytes, int part_bytes, int table_bytes) {
  const int att_bytes = p.D == 64 ? (int)sizeof(AttScratch<64>) : (int)sizeof(AttScratch<128>);
  static_assert(sizeof(AttScratch<64>) >= (kNT / 16 * 64 + 2 * (kNT / 16)) * 4 && sizeof(AttScratch<128>) >= (kNT / 32 * 128 + 2 * (kNT / 32)) * 4,
                "merge_head works in the same scratch");
  const bool shared = xin_bytes >= att_bytes;
  p.off_xin = kHeaderBytes + resid_bytes;
  p.off_xsum = p.off_xin + xin_bytes;
  p.off_part = p.off_xsum + xsum_bytes;
  p.off_table = p.off_part + part_bytes;
  p.off_att = shared ? p.off_xin : p.off_table + table_bytes;
  p.off_ring = p.off_table + table_bytes + (shared ? 0 : (att_bytes + 127) / 128 * 128);
  return (size_t)p.off_ring;
}
int decode_step_threads() { return kThreads; }
int decode_step_max_stages() { return kMaxStages; }
int decode_step_consumer_warps() { return kNCW; }
int decode_step_max_kv_tokens() { return kMaxKvTokens; }

// Whether a context of up to ctx_cap tokens can call for slices that are merged while staging.
static bool decode_step_staged(const StepParams& p, int ctx_cap) {
  return p.att_max <= 1 && p.att_slices > 1 && ctx_cap >= B200_STEP_STAGED_MIN;
}

cudaError_t decode_step_launch(const StepParams& p, int ctx_cap, int grid, size_t smem, cudaStream_t st) {
  const int kmax = p.H > p.I ? (p.H > p.n_att ? p.H : p.n_att) : (p.I > p.n_att ? p.I : p.n_att);
  const bool staged = decode_step_staged(p, ctx_cap);
  const bool wide = !staged && kmax > 128 * kNCW * kWideUnits;
  auto kern = p.D == 64 ? (staged ? decode_step_kernel<64, false, true> : wide ? decode_step_kernel<64, true, false> : decode_step_kernel<64, false, false>)
                        : (staged ? decode_step_kernel<128, false, true> : wide ? decode_step_kernel<128, true, false> : decode_step_kernel<128, false, false>);
  static size_t allowed[6][kMaxDevices] = {};
  const cudaError_t e = allow_dynamic_smem(kern, smem, allowed[3 * (p.D == 128) + 2 * staged + wide]);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;   // all CTAs co-resident, or the launch is refused
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

}  // namespace b200
