// W4A16 dequantize-GEMM for up to 64 tokens (the memory-bound decode regime), group-sum form, sm_100a:
//   C[m, n] = cast( sum_g s[g, n] * ( sum_{k in g} float(A[m, k]) * (q[n, k] - zero) ) )
// i.e. the group scale multiplies the group's fp32 partial sum instead of every weight.  With one-hot
// activations this equals half(q - zero) * s bit for bit (the fp32 product of two f16 values is exact
// and is rounded once, to the output type); in general it differs from scaling each weight in f16 first
// only by that product's own rounding (2^-11 relative per term), well inside the operator's tolerance.
//
// What bounds these shapes is not memory but the number of instructions and hand-overs an SM spends per 16 KB slab of
// packed weights (a slab's HBM time is about 700 cycles per SM), so the kernel is built to spend few:
//  - Conversion in nine instructions per eight weights: masking a nibble and setting an exponent around it in one lop3, so
//    that q in the low bits of 1024 is 1024 + q and q above the low four bits of 64 is 64 + q, and one f16 subtraction of
//    1024 + zero or 64 + zero: (q - zero), exactly.  (Leaving the zero point to the end - masked nibbles as subnormals, five
//    instructions, and one more MMA that takes zero * sum(A) off the accumulator - is no faster: 16 x 4096 x 4096 9.4 us
//    against 8.5, 32 of them in one call 73.4 / 71.3, 1, 32 and 64 tokens of 8192 x 28672 25.2 / 24.9, 31.4 / 29.8 and
//    40.8 / 40.5; only raw nibbles, 64 tokens, 38.0 / 39.5.  And a large
//    activation at a weight equal to zero then costs all other terms of the half their low bits: 18 to 400 times the
//    bound of test_large_activations_at_the_zero_point; an infinite one makes the difference NaN.)
//  - Activations are laid out by the pre-pass in the kernel's K order, so that a stage is one copy.  (Four, one for every 64 k, which
//    could leave out the rows beyond M without a tensor map, are more than the producer gets to issue: one token of 8192 x 28672
//    29.9 us instead of 26.5.)
//  - All hand-overs are by whole slabs; one commit per slab signals one barrier that the weight stage, the activation
//    stage and the accumulators share; the group scales arrive with the packed bytes and need no barrier of their own.
//
// Structure (persistent; the K slabs of the tiles are dealt to the CTAs, see W4HybridIter):
//   warp 0        TMA: packed weights [128 rows x 128 B] per slab into the raw ring, the slab's scale (and zero) rows
//   warp 1        TMA: prepared activations
//   warps 2, 3    tcgen05.mma kind::f16 issuers (A = weights from tensor memory, B = activations from shared memory):
//                 issuer w takes the slabs i with i % 2 == w, each of the two halves into its own accumulator
//   warps 4..11   drain: tcgen05.ld of a half's accumulator, fp32 FMA with the half's scale into register sums, in two sets of
//                 four warps (one per 32 rows); then the tile write or the split-K hand-over.  16 tokens: set e takes the
//                 slabs of parity e and the sets add their sums at a segment's end.  32 and 64 tokens: set e takes half of
//                 the tokens of every slab
//   warps 12..19  dequant: set s (four warps, one per 32 rows) converts the slabs of parity s
//   warps 20..23  split-K hand-overs
// Tensor memory: NS slots of two accumulators of MT columns + WS stages of 128 columns of converted weights.
//
// Every wait is bounded: after a number of failed mbarrier.try_wait attempts (each suspends the thread
// for a few microseconds) derived from the caller's limit, the wait stores its role code in a CTA-wide
// abort word and sets the thread's `fail` flag; all other waits of the CTA see the abort word in their
// slow path and give up too.  `fail` never steers a warp's control flow lane by lane (the tcgen05 ld /
// st / fence instructions need the whole warp): roles vote on it at coarse points, stop, and the kernel
// drains, frees its tensor memory, reports the code in the status word and returns.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "w4a16.cuh"

namespace qg {

constexpr int W4G_FIRST_MMA_WARP = 2;
constexpr int W4G_MMA_WARPS = 2;
constexpr int W4G_FIRST_EPI_WARP = 4;
constexpr int W4G_EPI_WARPS = 8;
constexpr int W4G_FIRST_DQ_WARP = W4G_FIRST_EPI_WARP + W4G_EPI_WARPS;  // 12
constexpr int W4G_DQ_SETS = 2;      // sets of four dequant warps
constexpr int W4G_FIN_WARP = W4G_FIRST_DQ_WARP + 4 * W4G_DQ_SETS;  // 20..23: split-K hand-overs
constexpr int W4G_THREADS = (W4G_FIN_WARP + 4) * 32;               // 768: at most 80 registers per thread
constexpr int W4G_SLAB_COLS = 128;  // tensor-memory columns of a converted slab
constexpr int W4G_SC_BYTES = 512;   // a slab's scales: up to two rows of 128 halves
constexpr int W4G_BARS = 8;         // barriers of a ring (whatever the number of data stages behind it), indexed by slab % 8

// Byte offsets of the barriers (8 bytes each) and control words from the start of the barrier block.
constexpr int W4G_RAW_FULL = 0;       // [8] a slab's packed weights (and scale rows) have landed
constexpr int W4G_RAW_EMPTY = 64;     // [8] its set has them in registers
constexpr int W4G_A_FULL = 128;       // [8] its activations have landed
constexpr int W4G_W_FULL = 192;       // [8] its converted weights are in tensor memory
constexpr int W4G_DONE = 256;         // [8] its MMAs have completed
constexpr int W4G_ACC_EMPTY = 320;    // [<= 4] an accumulator slot has been drained
constexpr int W4G_W_FULL0 = 352;      // [8] halves as steps (64 tokens): the first half's converted weights,
constexpr int W4G_DONE0 = 416;        // [8]   and its MMAs
constexpr int W4G_PART_READY = 480;   // [2] the CTA's (at most two) partial tiles: its sums are in the scratch buffer
constexpr int W4G_DRAIN = 496;
constexpr int W4G_PART_FULL = 504;    // SMALL form, in the cluster's first CTA: the other CTAs' sums have arrived
constexpr int W4G_TMEM_SLOT = 512;
constexpr int W4G_CTL = 520;          // u32 abort word (0, or the role code of the first wait that gave up), u32 max tries
constexpr int W4G_FIN_WORD = 528;     // u32[2], one per partial tile: its arrival number
constexpr int W4G_SMALL_MAX_SLABS = 4;  // SMALL form: slabs per CTA (stages 4.. of the raw ring receive the other CTAs' sums)

// Bytes of one prepared activation half: MT rows x 128 k of f16 (two 128-byte-swizzled blocks of 64 k).
__host__ __device__ constexpr int w4g_half_bytes(int mt) { return mt * 256; }

template <int MT, bool ZT = false>
struct W4GCfg {
  static_assert(MT == 16 || MT == 32 || MT == 64, "token tile");
  // Rings, in slabs.  64 KB of raw (packed) weights in flight per SM already stream at full speed.
  static constexpr int RS = (MT == 16) ? 8 : 4;           // raw weights, 16 KB each
  static constexpr int AS = (MT == 16) ? 4 : (MT == 32 ? 7 : 4);  // activations
  static constexpr int WS = (MT <= 32) ? 3 : 2;           // converted weights (tensor memory)
  static constexpr int NS = (MT == 16) ? 4 : 2;           // accumulator slots of two halves (even: a slot belongs to one set)
  static constexpr int SS = (RS == 8) ? 32 : 16;          // scale rows (see the note at the weight producer)
  static constexpr int A_HALF = w4g_half_bytes(MT);
  static constexpr int A_BYTES = 2 * A_HALF;              // one slab
  static constexpr int TMEM_COLS = 512;
  static constexpr int BAR_BYTES = 576;
  // 64 tokens: tensor memory holds two slabs of converted weights only, so the hand-over to the MMAs and back is by
  // halves - otherwise both sets convert while the tensor pipe idles and then both wait for it.
  static constexpr bool HALVES = MT == 64;
  // Above 16 tokens each drain set takes half of the tokens of every slab, so that a thread has one load of a half's sums to
  // wait for instead of a chain of them (64 tokens, 8192 x 28672: 41.2 -> 36.9 us; back to back for seconds, where the power
  // limit sets the clock, 48.3 -> 45.1; 48 tokens, 8192 x 8192, zeros tensor 22.4 -> 19.4).  Giving accumulators and converted
  // weights back half by half, in rings of 3 + 5 or 4 + 4 halves, was slower: 51.1 and 47.7.
  static constexpr bool BY_TOKENS = MT > 16;
  static constexpr int DT = BY_TOKENS ? MT / 2 : MT;      // tokens a drain thread accumulates
  static constexpr int DRAIN_WARPS = BY_TOKENS ? W4G_EPI_WARPS : W4G_EPI_WARPS / 2;  // that read a slab's accumulators
  static constexpr int XBUF_BYTES = BY_TOKENS ? 0 : MT * W4_BN * 4;  // the second drain set's sums of one segment
  static constexpr int SMEM_BYTES = RS * W4_RAW_PACKED + AS * A_BYTES + SS * W4G_SC_BYTES + (ZT ? RS * W4G_SC_BYTES : 0) +
                                    XBUF_BYTES + BAR_BYTES + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory of a CTA");
  static_assert(NS * 2 * MT + WS * W4G_SLAB_COLS <= 512 && (RS & (RS - 1)) == 0 && NS % 2 == 0 && AS < W4G_BARS, "layout");
};

// Debug hook for the bounded-wait test: when non-zero, the MMA issuers do not signal the completion of
// the last slab of the launch, so the drain warps' wait for it runs out.  Nothing else is affected:
// every copy lands, every other barrier completes, the kernel frees its tensor memory and returns.
struct W4GDebug {
  int withhold_last_commit;  // 1: as described above (two-launch form); 2: the single-launch form's cluster signal
};

// ---- lean primitives on shared-space addresses ------------------------------------------------------
// Bounded wait on the barrier at [base + OFF].  Fast path: one try_wait and one branch.  Slow path (the
// phase was not complete): poll; every failed try_wait has suspended the thread for a few microseconds,
// so the abort word and the attempt counter (both in the control block at `ctl`) are only looked at there.
template <int OFF, int CODE>
__device__ __forceinline__ void w4g_wait(uint32_t base, uint32_t parity, uint32_t ctl, uint32_t& fail) {
  asm volatile(
      "{\n\t"
      ".reg .pred p, q;\n\t"
      ".reg .u32 n, t;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1+%4], %2;\n\t"
      "@p bra W4G_DONE;\n\t"
      "ld.shared.u32 n, [%3+4];\n"
      "W4G_LOOP:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1+%4], %2;\n\t"
      "@p bra W4G_DONE;\n\t"
      "ld.volatile.shared.u32 t, [%3];\n\t"
      "setp.ne.u32 q, t, 0;\n\t"
      "@q bra W4G_FAIL;\n\t"
      "sub.u32 n, n, 1;\n\t"
      "setp.ne.u32 q, n, 0;\n\t"
      "@q bra W4G_LOOP;\n\t"
      "mov.u32 t, %5;\n\t"
      "st.volatile.shared.u32 [%3], t;\n"
      "W4G_FAIL:\n\t"
      "mov.u32 %0, 1;\n"
      "W4G_DONE:\n\t"
      "}"
      : "+r"(fail)
      : "r"(base), "r"(parity), "r"(ctl), "n"(OFF), "n"(CODE)
      : "memory");
}
template <int OFF>
__device__ __forceinline__ void w4g_arrive(uint32_t base) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0+%1];" ::"r"(base), "n"(OFF) : "memory");
}
template <int OFF>
__device__ __forceinline__ uint4 w4g_lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4+%5];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr), "n"(OFF));
  return v;
}
// One lane of the (converged) warp, chosen by the hardware.  Code under `if (w4g_elect_one())` is known to the
// compiler to run in exactly one lane, which lets it issue tcgen05.mma / commit / TMA instructions with their
// operands in uniform registers directly: measured 68 instead of 130-160 instructions, and 420 instead of 800-900
// cycles, for the eight MMAs and three commits of a half compared with `if (lane == 0)` or per-lane predicates.
__device__ __forceinline__ bool w4g_elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ void w4g_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Two fp32 FMAs in one instruction (d0 += a0 * s, d1 += a1 * s), each rounded exactly like fmaf: the drain warps'
// instruction streams are serial chains, so halving their FMA count shortens the chain.
__device__ __forceinline__ void w4g_fma2(float& d0, float& d1, uint32_t a0, uint32_t a1, float s) {
  asm("{\n\t"
      ".reg .b64 ra, rb, rc;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rb, {%4, %4};\n\t"
      "mov.b64 rc, {%0, %1};\n\t"
      "fma.rn.f32x2 rc, ra, rb, rc;\n\t"
      "mov.b64 {%0, %1}, rc;\n\t"
      "}"
      : "+f"(d0), "+f"(d1)
      : "r"(a0), "r"(a1), "f"(s));
}
// Named barrier of the eight drain warps.
__device__ __forceinline__ void w4g_epi_bar() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// The segments of a CTA: those of its stream-K range, then its whole tiles (first_dp, first_dp + stride, ...).
struct W4HybridIter {
  W4SegIter sk;
  int next_dp, dp_left, stride, KS;
  __device__ __forceinline__ bool next(int& tile, int& ks0, int& ks1) {
    if (sk.next(tile, ks0, ks1)) return true;
    if (dp_left <= 0) return false;
    tile = next_dp;
    ks0 = 0;
    ks1 = KS;
    next_dp += stride;
    --dp_left;
    return true;
  }
  __device__ __forceinline__ bool done() const { return sk.item >= sk.end && dp_left <= 0; }
};


// ---- prepared activations ---------------------------------------------------------------------------------------
// A 32-k chunk of a row becomes two groups of 16 f16 values: those whose weights the conversion finds in the low nibbles
// of the bytes it masks, then those in the high ones.  Word w of a packed 16-byte chunk holds elements 8 w .. 8 w + 7:
// low 8 w + {0, 4, 2, 6}, high 8 w + {1, 5, 3, 7}.
// v: the eight values of word w as four f16x2 words (0 1)(2 3)(4 5)(6 7) -> lo, hi: two f16x2 words each.
__device__ __forceinline__ void w4g_split_word(const uint4& v, uint2& lo, uint2& hi) {
  lo = make_uint2(__byte_perm(v.x, v.z, 0x5410), __byte_perm(v.y, v.w, 0x5410));
  hi = make_uint2(__byte_perm(v.x, v.z, 0x7632), __byte_perm(v.y, v.w, 0x7632));
}
__device__ __forceinline__ uint4 w4g_to_f16(uint4 v, bool is_bf16) {
  if (is_bf16) {
    v.x = w4_bf16x2_to_f16x2(v.x);
    v.y = w4_bf16x2_to_f16x2(v.y);
    v.z = w4_bf16x2_to_f16x2(v.z);
    v.w = w4_bf16x2_to_f16x2(v.w);
  }
  return v;
}
// Byte offset of 16-byte piece j (0..15) of row r inside a half of an activation stage: 64-k block j / 8, 128-byte swizzle.
template <int MT>
__device__ __forceinline__ uint32_t w4g_a_offset(int r, int j) {
  return (uint32_t)((j >> 3) * (MT * 128) + r * 128 + (((j & 7) ^ (r & 7)) << 4));
}

// One 32-k chunk (chunk c of four) of row r: four 16-byte loads already in v -> a half of a stage (single-launch form).
template <int MT>
__device__ __forceinline__ void w4g_emit_chunk(uint8_t* dst, int r, int c, const uint4 (&v)[4]) {
  uint2 lo[4], hi[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) w4g_split_word(v[w], lo[w], hi[w]);
  *reinterpret_cast<uint4*>(dst + w4g_a_offset<MT>(r, 4 * c + 0)) = make_uint4(lo[0].x, lo[0].y, lo[1].x, lo[1].y);
  *reinterpret_cast<uint4*>(dst + w4g_a_offset<MT>(r, 4 * c + 1)) = make_uint4(lo[2].x, lo[2].y, lo[3].x, lo[3].y);
  *reinterpret_cast<uint4*>(dst + w4g_a_offset<MT>(r, 4 * c + 2)) = make_uint4(hi[0].x, hi[0].y, hi[1].x, hi[1].y);
  *reinterpret_cast<uint4*>(dst + w4g_a_offset<MT>(r, 4 * c + 3)) = make_uint4(hi[2].x, hi[2].y, hi[3].x, hi[3].y);
}

// Pre-pass: activations [batch, M, K] (f16 or bf16) -> f16 [batch][64-k block][M][64] in the kernel's K order, whose blocks a tiled
// copy lays out as an activation stage wants them, rows beyond M zero.  (Rows that are left as they were reach nobody's sums but
// cost power: one token of 8192 x 28672 29.7 us for seconds instead of 28.1.)  A warp takes the 256 k of a slab of one
// row at a time, eight values a lane, `per` of them in flight.  k beyond K are zero.  Block 0 also zeroes the split-K arrival
// counters, so every call starts from clean counters whatever an earlier (possibly aborted) call left in the scratch.
// What bounds it is latency, between the end of the kernel in front and the GEMM kernel's first MMA, so all of its blocks should
// be waiting on an SM each when that kernel ends.  Behind another call of this operator, whose CTAs hold every SM, that takes
// blocks that fit beside a CTA of the GEMM kernel - 128 threads of 32 registers, what its 768 x 80 leave of the register file, and
// what its shared memory leaves - and no more of them than SMs (but see launch_w4g_prepare).  More blocks than that (one for every
// 128 chunks of 32 k of all MT rows) waited for the first SMs to become free, filled these, 16 to an SM, and kept the next call's
// GEMM CTAs off them for up to 10 us: 32 x 16 x 4096 x 4096 61.9 -> 59.2 us, 11 x 2 x 4352 x 1344 18.3 -> 14.4, 16 x 48 x 4096 x 2048 32.1 -> 28.3.
// LANDING: the values in flight wait in shared memory, since 32 registers hold two; with one or two the way through shared
// memory is the longer one (2 x 1280 x 14752 5.70 us, 5.60 without).
constexpr int W4G_PREP_THREADS = 128;
constexpr int W4G_PREP_REGS = 2;      // (row, slab) in flight per warp in registers,
constexpr int W4G_PREP_LANDING = 10;  // in shared memory: 20 KB, what a CTA of the 64-token kernel leaves
__device__ __forceinline__ void w4g_prep_emit(uint8_t* out, uint4 v, bool is_bf16, int M, int b, int m, int KS, int ks, int lane) {
  const int w = lane & 3, piece = (lane & 4) + (w >> 1);  // word w of the block's 32-k chunk (lane / 4) % 2
  uint2 lo, hi;
  w4g_split_word(w4g_to_f16(v, is_bf16), lo, hi);
  uint8_t* dst = out + ((((size_t)b * KS + ks) * 4 + (lane >> 3)) * M + m) * 128 + piece * 16 + (w & 1) * 8;
  *reinterpret_cast<uint2*>(dst) = lo;
  *reinterpret_cast<uint2*>(dst + 32) = hi;
}
template <bool LANDING>
__global__ void __launch_bounds__(W4G_PREP_THREADS, 16)
w4g_prepare_activations(const uint4* in, uint8_t* __restrict__ out, int rows, int M, int K, int KS, int is_bf16, int per,
                        uint4* __restrict__ counters, int n_counters) {
  pdl_launch_dependents();  // the GEMM kernel behind may set up and start streaming weights meanwhile
  const int lane = threadIdx.x & 31, warp = (int)(blockIdx.x * (W4G_PREP_THREADS / 32) + (threadIdx.x >> 5));
  const int first = per * warp, step = per * (int)gridDim.x * (W4G_PREP_THREADS / 32);
  int row = first / KS, ks = first - row * KS;  // row: of all problems'
  int b0 = row / M, m0 = row - b0 * M;
  pdl_wait();  // the kernel in front (another call's GEMM, which lets its dependents start early) is done
  auto src = [&](int r, int k) { return in + ((size_t)r * (size_t)K + k * W4_SLAB_K) / 8 + lane; };  // K is a multiple of 32
  auto in_row = [&](int k) { return k * W4_SLAB_K + lane * 8 < K; };
  while (row < rows) {
    int r = row, k = ks, b = b0, m = m0;
    auto next = [&]() {
      if (++k == KS) {
        k = 0;
        ++r;
        if (++m == M) { m = 0; ++b; }
      }
    };
    if constexpr (LANDING) {
      __shared__ uint4 landing[W4G_PREP_LANDING * W4G_PREP_THREADS];
      const uint4* mine = landing + threadIdx.x;  // a thread reads only what it has copied itself
      const int n = min(per, (rows - row) * KS - ks);
      for (int u = 0; u < n; ++u) {
        if (in_row(k)) cp_async16(smem_u32(mine + u * W4G_PREP_THREADS), src(r, k));
        if (++k == KS) { k = 0; ++r; }
      }
      cp_async_wait();
      r = row;
      k = ks;
#pragma unroll 1
      for (int u = 0; u < n; ++u) {
        w4g_prep_emit(out, in_row(k) ? mine[u * W4G_PREP_THREADS] : make_uint4(0u, 0u, 0u, 0u), is_bf16 != 0, M, b, m, KS, k, lane);
        next();
      }
    } else {
      uint4 v[W4G_PREP_REGS];
#pragma unroll
      for (int u = 0; u < W4G_PREP_REGS; ++u) {
        v[u] = u < per && r < rows && in_row(k) ? ld_written(src(r, k)) : make_uint4(0u, 0u, 0u, 0u);
        if (++k == KS) { k = 0; ++r; }
      }
      r = row;
      k = ks;
#pragma unroll
      for (int u = 0; u < W4G_PREP_REGS; ++u) {
        if (u < per && r < rows) w4g_prep_emit(out, v[u], is_bf16 != 0, M, b, m, KS, k, lane);
        next();
      }
    }
    ks += step;
    row += ks / KS;
    ks %= KS;
    b0 = row / M;
    m0 = row - b0 * M;
  }
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < n_counters / 4; i += W4G_PREP_THREADS) counters[i] = make_uint4(0u, 0u, 0u, 0u);
}

// Sixteen packed bytes (32 weights) -> eight f16x2 words of the low nibbles' q - zero, then eight of the high ones', K order
// as in w4g_split_word.  lo_sub = 1024 + zero, hi_sub = 64 + zero (both f16x2): every sum and difference here is exact.
// Interleaved layout (nibbles 0 2 4 6 | 1 3 5 7): three more instructions per eight weights, the same words, so that both
// layouts give the same sums bit for bit.
__device__ __forceinline__ uint32_t w4g_lo2(uint32_t x, uint32_t lo_sub) {
  uint32_t o;
  asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(o) : "r"(x));
  asm("sub.rn.f16x2 %0, %0, %1;" : "+r"(o) : "r"(lo_sub));
  return o;
}
__device__ __forceinline__ uint32_t w4g_hi2(uint32_t x, uint32_t hi_sub) {
  uint32_t o;
  asm("lop3.b32 %0, %1, 0x00f000f0, 0x54005400, 0xea;" : "=r"(o) : "r"(x));
  asm("sub.rn.f16x2 %0, %0, %1;" : "+r"(o) : "r"(hi_sub));
  return o;
}
template <bool INTERLEAVED>
__device__ __forceinline__ void w4g_convert(const uint4& v, uint32_t lo_sub, uint32_t hi_sub, uint32_t (&o)[16]) {
  const uint32_t x[4] = {v.x, v.y, v.z, v.w};
  if constexpr (!INTERLEAVED) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t y = x[w] >> 8;
      o[2 * w] = w4g_lo2(x[w], lo_sub);
      o[2 * w + 1] = w4g_lo2(y, lo_sub);
      o[8 + 2 * w] = w4g_hi2(x[w], hi_sub);
      o[8 + 2 * w + 1] = w4g_hi2(y, hi_sub);
    }
  } else {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t ev = __byte_perm(x[w], 0u, 0x4140), od = __byte_perm(x[w], 0u, 0x4342);  // (0 2 | 4 6), (1 3 | 5 7)
      o[2 * w] = w4g_lo2(ev, lo_sub);
      o[2 * w + 1] = w4g_lo2(ev >> 4, lo_sub);
      o[8 + 2 * w] = w4g_hi2(od << 4, hi_sub);
      o[8 + 2 * w + 1] = w4g_hi2(od, hi_sub);
    }
  }
}
// What w4g_convert takes for a zero point z, an integer as f16 in both halves of z2: 1024 + z and 64 + z.
__device__ __forceinline__ uint2 w4g_zero_subs(uint32_t z2) {
  uint2 s;
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(s.x) : "r"(0x64006400u), "r"(z2));
  asm("add.rn.f16x2 %0, %1, %2;" : "=r"(s.y) : "r"(0x54005400u), "r"(z2));
  return s;
}

// The sums of tokens m0 .. m0 + MT - 1 (those below M) of output feature n.
template <int MT, bool OUT_BF16, bool GATHER>
__device__ __forceinline__ void w4g_store_tile(const W4A16Params& p, int b, int m0, int n, const float (&sum)[MT]) {
  uint16_t* Cout = reinterpret_cast<uint16_t*>(p.C) + (size_t)b * p.M * p.N;
#pragma unroll
  for (int j = 0; j < MT; ++j)
    if (m0 + j < p.M) w4_store_out<OUT_BF16, GATHER>(p, Cout, m0 + j, n, sum[j]);
}

// GATHER = true is the gathered form (several destination buffers, see W4A16Params::c_dst); it is a separate
// instantiation because the destination loop in the store path costs the plain kernel registers.
// ZT = true: one integer zero point per (group, output feature) instead of the scalar one - the zeros tensor
// [K/g, N] f16 of zero mode "quantized" (tilelang/quantize/lop3.py:325-358: (q - qz) * s with the subtraction
// exact).  The weight producer fetches the slab's zero rows (through tmZ, laid out like the scale rows) into a ring
// that shares the packed weights' stages and barriers, and a dequant thread takes its row's zero point from there.
// SMALL = true (16-token tile): the single-launch form for problems of a few slabs per CTA.  The kernel is launched in
// clusters of C = KS / (slabs per CTA) CTAs, one tile per cluster, CTA r taking the r-th K range; there is no pre-pass
// and no scratch memory:
//  - the drain warps first fetch the CTA's own piece of the activations straight from the caller's tensor and write the
//    stages as the copies of what the pre-pass makes would have;
//  - at the end CTAs 1 .. C-1 write their sums through distributed shared memory into the unused upper half of the
//    first CTA's raw ring, and the first CTA adds them in rank order and writes the tile - no counters, no partial
//    sums in global memory, the same fixed summation order on every run.
template <int MT, bool OUT_BF16, bool GATHER = false, bool ZT = false, bool SMALL = false>
__global__ void __launch_bounds__(W4G_THREADS, 1)
w4a16_gs_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS,
                const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmA, const __grid_constant__ W4A16Params p,
                const W4GDebug dbg) {
  using Cfg = W4GCfg<MT, ZT>;
  constexpr int RS = Cfg::RS;
  constexpr int AS = Cfg::AS;
  constexpr int NS = Cfg::NS;
  constexpr int WS = Cfg::WS;
  static_assert(RS <= 8 && NS <= 4, "barrier block layout");
  static_assert(!SMALL || (MT == 16 && !GATHER && !ZT), "the single-launch form: 16-token tile, one destination, scalar zero");
  // The next call's pre-pass (a programmatic dependent) may become resident now; it waits for this whole grid before
  // it touches anything, and the GEMM kernel behind it only reads weights and scales until that pre-pass is done.
  pdl_launch_dependents();

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw_base = smem;
  uint8_t* a_base = raw_base + RS * W4_RAW_PACKED;
  uint8_t* sc_base = a_base + AS * Cfg::A_BYTES;
  uint8_t* z_base = sc_base + Cfg::SS * W4G_SC_BYTES;     // zero rows, one 512-byte stage per raw stage (ZT only)
  float* xbuf = reinterpret_cast<float*>(z_base + (ZT ? RS * W4G_SC_BYTES : 0));
  uint8_t* bar_block = reinterpret_cast<uint8_t*>(xbuf) + Cfg::XBUF_BYTES;
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(bar_block + W4G_RAW_FULL);
  uint64_t* a_full = reinterpret_cast<uint64_t*>(bar_block + W4G_A_FULL);
  uint64_t* drain = reinterpret_cast<uint64_t*>(bar_block + W4G_DRAIN);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_block + W4G_TMEM_SLOT);
  volatile uint32_t* ctl_words = reinterpret_cast<uint32_t*>(bar_block + W4G_CTL);  // [0] abort word, [1] max tries

  // a warp index the compiler can prove uniform, so that everything derived from it may live in uniform registers
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;

  // One thread per barrier slot sets it up (the block is a dense array of 8-byte slots).
  if (threadIdx.x <= W4G_PART_FULL / 8) {
    const int off = 8 * (int)threadIdx.x;
    int count = 0;                                          // 0: unused slot
    if (off < W4G_RAW_EMPTY) count = 1;
    else if (off < W4G_A_FULL) count = 4;      // the four dequant warps of the slab's set
    else if (off < W4G_W_FULL) count = 1;
    else if (off < W4G_DONE) count = 4;
    else if (off < W4G_ACC_EMPTY) count = 1;
    else if (off < W4G_W_FULL0) count = Cfg::DRAIN_WARPS;
    else if (off < W4G_DONE0) count = 4;
    else if (off < W4G_PART_READY) count = 1;
    else if (off < W4G_DRAIN) count = Cfg::DRAIN_WARPS;
    else if (off < W4G_PART_FULL) count = W4G_MMA_WARPS;
    else if (SMALL) count = max((int)cluster_nctarank() - 1, 1);
    if (count > 0) mbar_init(reinterpret_cast<uint64_t*>(bar_block + off), (uint32_t)count);
    fence_barrier_init();
  }
  if (threadIdx.x == 64) {
    ctl_words[0] = 0;
    // a failed try_wait has suspended the thread for roughly 2 us or longer
    ctl_words[1] = (uint32_t)(p.wait_limit_ns >> 11) + 2u;
    tma_prefetch_desc(&tmW);
    if (p.has_scales) tma_prefetch_desc(&tmS);
    if (ZT) tma_prefetch_desc(&tmZ);
    if (!SMALL) tma_prefetch_desc(&tmA);
  }
  if (warp == W4G_FIRST_MMA_WARP + 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if constexpr (SMALL) cluster_sync_all();  // the first CTA's barrier exists before any other CTA of the cluster signals it
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_w = tmem_base + NS * 2 * MT;  // converted weights behind the accumulator ring
  const uint32_t bar0 = smem_u32(bar_block);
  const uint32_t ctl = bar0 + W4G_CTL;

  const int G = gridDim.x;
  const int cta = blockIdx.x;
  // Work split: the first p.sk_tiles tiles are cut stream-K fashion (their slabs dealt evenly to the CTAs as
  // contiguous ranges, partial tiles meeting through the scratch buffer); after its range CTA c takes the whole tiles
  // sk_tiles + c, sk_tiles + c + G, ...  The hand-overs of the partial tiles thus happen early, behind the following
  // tiles' work, and the launch ends with plain tile writes.
  const long long T = (long long)p.sk_tiles * p.KS;  // stream-K items
  // SMALL: cluster t takes tile t, its CTA r the slabs [r * per, (r + 1) * per) of it
  const int crank = SMALL ? (int)cluster_ctarank() : 0;
  const int csize = SMALL ? (int)cluster_nctarank() : 1;
  const int per = SMALL ? p.KS / csize : 0;
  const long long item0 = SMALL ? (long long)(cta / csize) * p.KS + (long long)crank * per : w4_range_begin(T, G, cta);
  const long long item1 = SMALL ? item0 + per : w4_range_begin(T, G, cta + 1);
  const int n_sk = (int)(item1 - item0);
  const int n_slabs = SMALL ? n_sk : n_sk + p.dp_rounds * p.KS;  // this CTA's slabs, numbered 0.. in processing order

  // 64 tokens: a drain thread holds 32 sums and 32 values on their way into them, a hand-over thread two contributors' values,
  // more than the 80 registers the block is launched with; the producers and issuers give theirs up (48 + 2 x 88 + 2 x 80 + 96 =
  // 6 x 80).
  if constexpr (MT == 64) {
    if (warp < W4G_FIRST_EPI_WARP) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    else if (warp >= W4G_FIN_WARP) asm volatile("setmaxnreg.inc.sync.aligned.u32 96;");
    else if (warp < W4G_FIRST_DQ_WARP) asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
  }
  if (warp < 2) {
    // ------------------------------------------------------------------ producers
    // One thread each.  A thread of this kernel gets to issue an instruction only every ten cycles or so, so what a
    // producer does per slab is kept to a few dozen instructions (a slab's HBM time is 700 cycles).
    if (lane == 0 && !(SMALL && warp == 1)) {
      int tile = n_sk > 0 ? (int)(item0 / p.KS) : p.sk_tiles + cta;
      int ks = n_sk > 0 ? (int)(item0 - (long long)tile * p.KS) : 0;
      int b, n0, m0;
      w4_tile_coords(p, tile, MT, b, n0, m0);
      uint32_t fail = 0;
      uint32_t issued_mask = 0, parity_mask = 0;
      int left = n_sk > 0 ? min(n_sk, p.KS - ks) : p.KS;  // slabs up to the next change of tile
      int i = 0;
      if (warp == 0) {
        // Packed weights, and with them - on the same barrier - the slab's scale rows, into a ring of their own that is SS
        // slabs deep.  Loading slab L means that slab L - RS is in registers, so (its set having stored its previous slab,
        // L - RS - 2) the MMAs up to slab L - RS - 2 - WS have completed, for which the drain warps have left the slot
        // NS slabs further back: a scale slot is rewritten only after it has been read, without a barrier, as long as
        // SS >= RS + WS + NS + 3.  A drain warp reads a scale only after the slab's MMAs, i.e. after this barrier.
        static_assert(Cfg::SS >= RS + WS + NS + 3, "scale ring");
        const uint32_t row_tx = (uint32_t)p.scale_rows * 256u;
        const uint32_t tx = W4_RAW_PACKED + (p.has_scales ? row_tx : 0u) + (ZT ? row_tx : 0u);
        const int spg = p.scale_rows == 2 ? 1 : (p.group + W4_SLAB_K - 1) / W4_SLAB_K;  // slabs per scale row (pair)
        const int row_step = p.scale_rows == 2 ? 2 : 1;
        int srow = (ks / spg) * row_step, in_group = ks % spg;
        int st = 0;
        uint32_t phase = 0;
        const uint64_t once = l2_policy_evict_first();
        while (i < n_slabs) {
          w4g_wait<W4G_RAW_EMPTY, ST_TIMEOUT_PRODUCER>(bar0 + 8 * st, phase ^ 1u, ctl, fail);
          if (fail) break;
          mbar_arrive_expect_tx(&raw_full[st], tx);
          tma_load_3d_hint(raw_base + st * W4_RAW_PACKED, &tmW, &raw_full[st], ks * (W4_SLAB_K / 2), n0, b, once);
          // scale rows of the slab: two when the groups are 128 wide, else the one row of the slab's group
          if (p.has_scales) tma_load_3d(sc_base + (i % Cfg::SS) * W4G_SC_BYTES, &tmS, &raw_full[st], n0, srow, b);
          if (ZT) tma_load_3d(z_base + st * W4G_SC_BYTES, &tmZ, &raw_full[st], n0, srow, b);
          issued_mask |= 1u << st;
          parity_mask = (parity_mask & ~(1u << st)) | (phase << st);
          if (++st == RS) { st = 0; phase ^= 1u; }
          ++i;
          ++ks;
          if (++in_group == spg) { in_group = 0; srow += row_step; }
          if (--left == 0) {  // the tile, or this CTA's share of it, is done
            tile = i == n_sk ? p.sk_tiles + cta : tile + (i < n_sk ? 1 : G);
            ks = srow = in_group = 0;
            left = i < n_sk ? min(n_sk - i, p.KS) : p.KS;
            w4_tile_coords(p, tile, MT, b, n0, m0);
          }
        }
      } else {
        int st = 0;
        // A CTA's first copies are what the kernel waits for when it has few slabs, so up to 16 tokens all that can be done for
        // them without the activations is done in front of the wait, and they are issued in one go behind it (1 x 1792 x 6288 9.5 ->
        // 8.9 us, 16 x 3584 x 4096 10.4 -> 8.8; 64 x 8192 x 28672 43.7 instead of 42.2).  Not with less than two slabs per CTA in
        // the mean, some with one and some with two, where all then hand over at once and it is slower (2 x 4864 x 1104 11.3 -> 12.1, 4 x
        // 3328 x 1696 9.9 -> 11.1, 8 x 4352 x 2048 9.8 -> 11.5; from there on 2 x 4352 x 2784 10.7 -> 9.5, 12 x 3328 x 3872 10.6 -> 9.4).
        if (MT == 16 && !SMALL && p.total_items >= 2 * G) {
          int first_z[AS];
          const int n_first = min(n_slabs, AS);
#pragma unroll
          for (int j = 0; j < AS; ++j) {
            first_z[j] = (b * p.KS + ks) * 4;
            if (j < n_first) {  // as below
              mbar_arrive_expect_tx(&a_full[j], Cfg::A_BYTES);
              ++ks;
              if (--left == 0) {
                tile = j + 1 == n_sk ? p.sk_tiles + cta : tile + (j + 1 < n_sk ? 1 : G);
                ks = 0;
                left = j + 1 < n_sk ? min(n_sk - (j + 1), p.KS) : p.KS;
                w4_tile_coords(p, tile, MT, b, n0, m0);
              }
            }
          }
          pdl_wait();
#pragma unroll
          for (int j = 0; j < AS; ++j)
            if (j < n_first) tma_load_3d(a_base + j * Cfg::A_BYTES, &tmA, &a_full[j], 0, 0, first_z[j]);
          issued_mask = (1u << n_first) - 1u;
          i = n_first;
          st = n_first == AS ? 0 : n_first;
        } else {
          pdl_wait();  // the prepared activations come from the pre-pass kernel in front of this one
        }
        while (i < n_slabs) {
          if (i >= AS)  // the slab that used this stage has been multiplied
            w4g_wait<W4G_DONE, ST_TIMEOUT_PRODUCER>(bar0 + 8 * ((i - AS) % W4G_BARS), (uint32_t)((i - AS) / W4G_BARS) & 1u, ctl, fail);
          if (fail) break;
          uint64_t* bar = &a_full[i % W4G_BARS];
          mbar_arrive_expect_tx(bar, Cfg::A_BYTES);
          tma_load_3d(a_base + st * Cfg::A_BYTES, &tmA, bar, 0, 0, (b * p.KS + ks) * 4);  // four blocks of 64 k, MT rows each
          issued_mask |= 1u << (i % W4G_BARS);
          parity_mask = (parity_mask & ~(1u << (i % W4G_BARS))) | (((uint32_t)(i / W4G_BARS) & 1u) << (i % W4G_BARS));
          if (++st == AS) st = 0;
          ++i;
          ++ks;
          if (--left == 0) {
            tile = i == n_sk ? p.sk_tiles + cta : tile + (i < n_sk ? 1 : G);
            ks = 0;
            left = i < n_sk ? min(n_sk - i, p.KS) : p.KS;
            w4_tile_coords(p, tile, MT, b, n0, m0);
          }
        }
      }
      if (fail) {  // wait (bounded) for the copies still in flight before the CTA may exit
        uint64_t* full = warp == 0 ? raw_full : a_full;
        for (int s = 0; s < 8; ++s) {
          if (!(issued_mask & (1u << s))) continue;
          const uint64_t t0 = global_timer_ns();
          while (!mbar_try_wait(&full[s], (parity_mask >> s) & 1u)) {
            if (global_timer_ns() - t0 > p.wait_limit_ns) {
              ctl_words[0] = ST_TIMEOUT_DRAIN;
              break;
            }
          }
        }
      }
    }
  } else if (warp < W4G_FIRST_EPI_WARP) {
    // ------------------------------------------------------------------ MMA issuers (warp-convergent)
    // Issuer w takes the slabs i with i % 2 == w: weight stage i % WS, activation stage i % AS, accumulator slot i % NS.
    const int w = warp - W4G_FIRST_MMA_WARP;
    constexpr uint32_t idesc = make_idesc(ACC_F32, FMT_F16, FMT_F16, 0, 0, W4_BN, MT);
    // K-major activation descriptor: the high word is constant, the low word holds the start address >> 4
    const uint64_t desc0 = make_desc_kmajor(smem_u32(a_base));
    const uint32_t desc_hi = (uint32_t)(desc0 >> 32);
    const uint32_t desc_lo0 = (uint32_t)desc0;
    const int withhold_i = (dbg.withhold_last_commit == 1 && cta == G - 1) ? n_slabs - 1 : -1;
    uint32_t fail = 0;
    int as = w % AS, ws = w % WS;
    for (int i = w; i < n_slabs; i += W4G_MMA_WARPS) {
      const int slot = i % NS;
      const uint32_t bi = bar0 + 8 * (i % W4G_BARS), par = (uint32_t)(i / W4G_BARS) & 1u;
      w4g_wait<W4G_ACC_EMPTY, ST_TIMEOUT_MMA>(bar0 + 8 * slot, ((uint32_t)(i / NS) & 1u) ^ 1u, ctl, fail);
      w4g_wait<W4G_A_FULL, ST_TIMEOUT_MMA>(bi, par, ctl, fail);
      const uint32_t d = tmem_base + slot * (2 * MT);
      const uint32_t tW = tmem_w + ws * W4G_SLAB_COLS;
      const uint32_t a_off = (uint32_t)((as * Cfg::A_BYTES) >> 4);
      auto issue_half = [&](auto half_) {
        constexpr int half = decltype(half_)::value;
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16) {
          const uint32_t off = (uint32_t)((half * Cfg::A_HALF + (k16 >> 2) * (MT * 128) + (k16 & 3) * 32) >> 4);
          const uint64_t bd = ((uint64_t)desc_hi << 32) | (uint64_t)(desc_lo0 + a_off + off);
          umma_f16_ts(d + half * MT, tW + half * (W4G_SLAB_COLS / 2) + k16 * 8, bd, idesc, k16 != 0 ? 1u : 0u);
        }
      };
      constexpr std::integral_constant<int, 0> H0{};
      constexpr std::integral_constant<int, 1> H1{};
      if constexpr (Cfg::HALVES) {
        w4g_wait<W4G_W_FULL0, ST_TIMEOUT_MMA>(bi, par, ctl, fail);
        tc_fence_after_sync();
        if (w4g_elect_one()) {
          issue_half(H0);
          w4g_commit(bi + W4G_DONE0);
        }
      }
      w4g_wait<W4G_W_FULL, ST_TIMEOUT_MMA>(bi, par, ctl, fail);
      tc_fence_after_sync();
      if (w4g_elect_one()) {
        if constexpr (!Cfg::HALVES) issue_half(H0);
        issue_half(H1);
        if (i != withhold_i) w4g_commit(bi + W4G_DONE);
      }
      as += W4G_MMA_WARPS;
      if (as >= AS) as -= AS;
      ws += W4G_MMA_WARPS;
      if (ws >= WS) ws -= WS;
      // `fail` is looked at rarely: what is issued after a wait that gave up stays inside this CTA's memories
      if ((i & 6) == 6) {
        fail = __any_sync(0xffffffffu, fail != 0) ? 1u : 0u;
        if (fail) break;
      }
    }
    // everything this warp issued has completed before the CTA frees its tensor memory
    if (w4g_elect_one()) w4g_commit(bar0 + W4G_DRAIN);
    if (w == 0 && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (!mbar_try_wait(drain, 0)) {
        if (global_timer_ns() - t0 > p.wait_limit_ns) break;
      }
    }
  } else if (warp < W4G_FIRST_DQ_WARP) {
    // ------------------------------------------------------------------ drain / epilogue
    const int e = (warp - W4G_FIRST_EPI_WARP) >> 2;  // drain set
    const int q = warp & 3;
    const int nl = q * 32 + lane;  // weight row inside the tile == TMEM lane
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t sc_addr0 = smem_u32(sc_base) + 2 * nl;
    const uint32_t sc_row1 = p.scale_rows == 2 ? 256u : 0u;  // the second half's scale row inside a stage
    const bool scaled = p.has_scales != 0;
    const bool lead = lane == 0;
    constexpr int DT = Cfg::DT;
    const int t_first = Cfg::BY_TOKENS ? e * DT : 0;  // first of this set's tokens
    if constexpr (!SMALL) pdl_wait();  // the arrival counters are zeroed by the pre-pass kernel in front of this one
    if constexpr (SMALL) {
      // this CTA's piece of the activations: rows m0 .. m0 + 15 (zero beyond M), k [256 * ks_first, 256 * (ks_first + per))
      const int tile_s = (int)(item0 / p.KS);
      const int ks_first = (int)(item0 - (long long)tile_s * p.KS);
      int bb, nn0, mm0;
      w4_tile_coords(p, tile_s, MT, bb, nn0, mm0);
      const int tid = (e * 4 + q) * 32 + lane;  // 0 .. 255
      const int units = MT * per * 8;           // 32-k chunks of this CTA: (half, row, chunk), a multiple of 128
      const uint4* src = reinterpret_cast<const uint4*>(p.A_raw) + ((size_t)bb * p.M) * (size_t)(p.K / 8);
      constexpr int PER_THREAD = MT * W4G_SMALL_MAX_SLABS * 8 / 256;  // at most two chunks per thread
      const uint4* ptr[PER_THREAD];
#pragma unroll
      for (int u = 0; u < PER_THREAD; ++u) {
        const int i = tid + 256 * u;
        const int c = i & 3, r = (i >> 2) % MT, hl = (i >> 2) / MT;
        const int k0 = ks_first * W4_SLAB_K + hl * 128 + c * 32;
        ptr[u] = (i < units && mm0 + r < p.M && k0 < p.K) ? src + (size_t)(mm0 + r) * (size_t)(p.K / 8) + k0 / 8 : nullptr;
      }
      pdl_wait();  // whatever is in front of this launch has finished: the activations may be read, the output written
      uint4 v[PER_THREAD][4];
#pragma unroll
      for (int u = 0; u < PER_THREAD; ++u)  // all loads first, so that their latencies overlap
#pragma unroll
        for (int k = 0; k < 4; ++k)
          v[u][k] = ptr[u] != nullptr ? __ldcg(ptr[u] + k) : make_uint4(0u, 0u, 0u, 0u);  // L2 is the point of coherence
#pragma unroll
      for (int u = 0; u < PER_THREAD; ++u) {
        const int i = tid + 256 * u;
        if (i < units) {  // warp-uniform: units is a multiple of 128
          const int c = i & 3, r = (i >> 2) % MT, hl = (i >> 2) / MT;
#pragma unroll
          for (int k = 0; k < 4; ++k) v[u][k] = w4g_to_f16(v[u][k], p.a_is_bf16 != 0);
          w4g_emit_chunk<MT>(a_base + hl * Cfg::A_HALF, r, c, v[u]);
        }
      }
      fence_proxy_async_smem();  // the MMAs read these stages through the async proxy
      w4g_epi_bar();
      if (tid == 0)
        for (int sl = 0; sl < per; ++sl) mbar_arrive(&a_full[sl]);
    }
    W4HybridIter seg{W4SegIter{item0, item1, p.KS}, p.sk_tiles + cta, SMALL ? 0 : p.dp_rounds, G, p.KS};
    int tile, ks0, ks1;
    uint32_t i_seg0 = 0;  // CTA-local index of the segment's first slab
    uint32_t fail = 0;
    int n_partial = 0;
    while (seg.next(tile, ks0, ks1)) {
      int b, n0, m0;
      w4_tile_coords(p, tile, MT, b, n0, m0);
      const int n = n0 + nl;
      const bool full_tile = (ks0 == 0 && ks1 == p.KS);
      const int my_slot = (ks1 < p.KS) ? 2 * cta + 1 : 2 * cta;
      const uint32_t i_end = i_seg0 + (uint32_t)(ks1 - ks0);
      float psum[DT];
#pragma unroll
      for (int m = 0; m < DT; ++m) psum[m] = 0.f;
      for (uint32_t i = Cfg::BY_TOKENS ? i_seg0 : i_seg0 + ((i_seg0 ^ (uint32_t)e) & 1u); i < i_end; i += Cfg::BY_TOKENS ? 1 : 2) {
        const uint32_t slot = i % NS;
        const uint32_t bs = bar0 + 8 * slot;
        const uint32_t bd = bar0 + 8 * (i % W4G_BARS), dpar = (i / W4G_BARS) & 1u;
        const uint32_t ta = tmem_base + lane_addr + slot * (2 * MT) + t_first;
        float s0 = 1.0f, s1 = 1.0f;
        auto load_scales = [&]() {  // after the slab's MMAs, see the note at the weight producer
          if (scaled) {
            uint16_t h0, h1;
            const uint32_t sa = sc_addr0 + (i % Cfg::SS) * W4G_SC_BYTES;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h0) : "r"(sa));
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(h1) : "r"(sa + sc_row1));
            s0 = __half2float(__ushort_as_half(h0));
            s1 = __half2float(__ushort_as_half(h1));
          }
        };
        auto release = [&]() {  // the accumulators are in registers
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lead) w4g_arrive<W4G_ACC_EMPTY>(bs);
        };
        if constexpr (DT == 16) {
          w4g_wait<W4G_DONE, ST_TIMEOUT_EPILOGUE>(bd, dpar, ctl, fail);
          tc_fence_after_sync();
          uint32_t r[32];  // the two halves
          if constexpr (MT == 16) {
            tmem_ld_32x32b_x32(ta, r);
          } else {
            tmem_ld_32x32b_x16(ta, reinterpret_cast<uint32_t(&)[16]>(r[0]));
            tmem_ld_32x32b_x16(ta + MT, reinterpret_cast<uint32_t(&)[16]>(r[16]));
          }
          load_scales();
          release();
#pragma unroll
          for (int m = 0; m < 16; m += 2) {
            w4g_fma2(psum[m], psum[m + 1], r[m], r[m + 1], s0);
            w4g_fma2(psum[m], psum[m + 1], r[16 + m], r[17 + m], s1);
          }
        } else {  // the first half's sums while the second half's MMAs run
          uint32_t r[32];
          w4g_wait<W4G_DONE0, ST_TIMEOUT_EPILOGUE>(bd, dpar, ctl, fail);
          tc_fence_after_sync();
          tmem_ld_32x32b_x32(ta, r);
          load_scales();
          tmem_ld_wait();
#pragma unroll
          for (int m = 0; m < 32; m += 2) w4g_fma2(psum[m], psum[m + 1], r[m], r[m + 1], s0);
          w4g_wait<W4G_DONE, ST_TIMEOUT_EPILOGUE>(bd, dpar, ctl, fail);
          tc_fence_after_sync();
          tmem_ld_32x32b_x32(ta + MT, r);
          release();
#pragma unroll
          for (int m = 0; m < 32; m += 2) w4g_fma2(psum[m], psum[m + 1], r[m], r[m + 1], s1);
        }
      }
      i_seg0 = i_end;
      // Segment end.  16 tokens: set 1 hands over its sums through shared memory, set 0 adds them.  The tile is written, or the
      // partial sums to the scratch buffer, where the split-K warps take over.  (A wait that gave up does not change the course
      // of events here: all waits of the CTA then give up quickly, and the status word says that C is unspecified.)
      float* xb = xbuf + nl;
      if constexpr (!Cfg::BY_TOKENS) {
        if (e == 1) {
#pragma unroll
          for (int j = 0; j < DT; ++j) xb[j * W4_BN] = psum[j];
        }
        w4g_epi_bar();
      }
      if constexpr (SMALL) {
        // One segment per CTA.  Set 0 holds the CTA's sums; CTAs 1 .. C-1 of the cluster write theirs into the first
        // CTA's landing area (the raw ring's stages 4 .. 7, never filled in this form) and signal it; the first CTA
        // adds them in rank order and writes the tile.
        if (e == 0) {
#pragma unroll
          for (int j = 0; j < DT; ++j) psum[j] += xb[j * W4_BN];
        }
        float* landing = reinterpret_cast<float*>(raw_base + W4G_SMALL_MAX_SLABS * W4_RAW_PACKED);  // [rank - 1][token][row]
        if (crank != 0) {
          if (e == 0 && __all_sync(0xffffffffu, fail == 0)) {
            const uint32_t dst = mapa_u32(smem_u32(landing + (size_t)(crank - 1) * (MT * W4_BN) + nl), 0);
#pragma unroll
            for (int j = 0; j < DT; ++j)
              asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)(j * W4_BN * 4)), "f"(psum[j]) : "memory");
            fence_acq_rel_cluster();
          }
          w4g_epi_bar();  // every thread's stores are issued and fenced before the one signal
          // (test hook, value 2: the last cluster's CTA 1 keeps its signal back, so that the first CTA's wait runs out)
          const bool withheld = dbg.withhold_last_commit == 2 && crank == 1 && cta / csize == G / csize - 1;
          if (warp == W4G_FIRST_EPI_WARP && lane == 0 && !fail && ctl_words[0] == 0 && !withheld)
            mbar_arrive_cluster(mapa_u32(bar0 + W4G_PART_FULL, 0));
        } else {
          bool got = true;
          if (csize > 1) {
            if (lane == 0) {
              const uint64_t t0 = global_timer_ns();
              while (!mbar_try_wait_cluster(reinterpret_cast<uint64_t*>(bar_block + W4G_PART_FULL), 0)) {
                if (ctl_words[0] != 0 || global_timer_ns() - t0 > p.wait_limit_ns) {
                  if (ctl_words[0] == 0) ctl_words[0] = ST_TIMEOUT_EPILOGUE;
                  got = false;
                  break;
                }
              }
            }
            got = __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0;
            fence_acq_rel_cluster();
          }
          if (got && e == 0 && !fail && n < p.N) {
            for (int c = 1; c < csize; ++c) {
              const float* src = landing + (size_t)(c - 1) * (MT * W4_BN) + nl;
#pragma unroll
              for (int j = 0; j < DT; ++j) psum[j] += src[j * W4_BN];
            }
            w4g_store_tile<MT, OUT_BF16, GATHER>(p, b, m0, n, psum);
          }
        }
        break;
      }
      if (Cfg::BY_TOKENS || e == 0) {
        if constexpr (!Cfg::BY_TOKENS) {
#pragma unroll
          for (int j = 0; j < DT; ++j) psum[j] += xb[j * W4_BN];
        }
        if (full_tile) {
          if (n < p.N) w4g_store_tile<DT, OUT_BF16, GATHER>(p, b, m0 + t_first, n, psum);
        } else {
          float* dst = p.ws_partials + (size_t)my_slot * (MT * W4_BN) + (size_t)t_first * W4_BN + nl;
#pragma unroll
          for (int j = 0; j < DT; ++j) dst[j * W4_BN] = psum[j];
          __syncwarp();
          if (lead) w4g_arrive<W4G_PART_READY>(bar0 + 8 * n_partial);
          ++n_partial;
        }
      }
      if constexpr (!Cfg::BY_TOKENS) w4g_epi_bar();  // set 0 has read the exchange buffer
    }
  } else if (warp >= W4G_FIN_WARP) {
    // ------------------------------------------------------------------ split-K hand-over
    // A tile that several CTAs share: each one's partial sums go to the scratch buffer and a counter tells the last
    // contributor (never by waiting), which adds them in a fixed order and writes the tile.  This chain of global-memory
    // round trips (fence, atomic, loads: 7 000 cycles when the drain warps ran it, with the pipeline standing still behind
    // them) is these four warps' alone; they take four tokens in turn, two contributors' at a time (20 x 7168 x 480, 28
    // contributors to a tile: 26.7 -> 16.7 us; a quarter of the tokens each, one contributor at a time and a 64-bit division
    // for every one of them was what it replaced).
    const int fw = warp - W4G_FIN_WARP;
    volatile uint32_t* fin_word = reinterpret_cast<uint32_t*>(bar_block + W4G_FIN_WORD);
    if constexpr (!SMALL) {
      pdl_wait();  // the arrival counters are zeroed by the pre-pass kernel in front of this one
      W4SegIter seg{item0, item1, p.KS};
      int tile, ks0, ks1;
      int n_partial = 0;
      uint32_t fail = 0;
      while (seg.next(tile, ks0, ks1)) {
        if (ks0 == 0 && ks1 == p.KS) continue;
        w4g_wait<W4G_PART_READY, ST_TIMEOUT_EPILOGUE>(bar0 + 8 * n_partial, 0u, ctl, fail);
        const long long first_item = (long long)tile * p.KS;
        const int b_first = w4_owner(T, G, first_item), b_last = w4_owner(T, G, first_item + p.KS - 1);
        if (fw == 0 && lane == 0) {
          __threadfence();
          fin_word[n_partial] = atomicAdd(p.ws_counters + b_first, 1u);
        }
        asm volatile("bar.sync 2, 128;" ::: "memory");
        const bool last = fin_word[n_partial] == (uint32_t)(b_last - b_first);
        ++n_partial;
        if (!last) continue;
        __threadfence();
        int b, n0, m0;
        w4_tile_coords(p, tile, MT, b, n0, m0);
        uint16_t* Cout = reinterpret_cast<uint16_t*>(p.C) + (size_t)b * p.M * p.N;
        const int n = n0 + 4 * lane;  // four rows of the tile per lane
        const int rows = min(MT, p.M - m0);
        // four tokens of two contributors in flight; of one at 33 .. 64 tokens: 64 x 8192 x 1024 27.6 us instead of 21.9, 64 x 8192 x
        // 4096 17.6 / 16.5, 2 x 58 x 2304 x 1008 20.6 / 17.8, 64 x 8192 x 28672 37.5 / 38.0 (32 bytes of spills either way)
        constexpr int RU = 4, CU = 2;
        // every contributor but the last one stops short of the tile's end: its partial tile is its second one (slot 2 c + 1)
        auto part = [&](int c, int m) {
          return reinterpret_cast<const float4*>(p.ws_partials + (size_t)(c == b_last ? 2 * c : 2 * c + 1) * (MT * W4_BN) +
                                                 (size_t)m * W4_BN) + lane;
        };
#pragma unroll 1
        for (int mb = RU * fw; mb < rows; mb += 4 * RU) {
          float4 sum[RU];
#pragma unroll
          for (int u = 0; u < RU; ++u) sum[u] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
          for (int c = b_first; c <= b_last; c += CU) {  // fixed order: results do not depend on arrival order
            float4 v[CU][RU];
#pragma unroll
            for (int i = 0; i < CU; ++i)
#pragma unroll
              for (int u = 0; u < RU; ++u)
                v[i][u] = c + i <= b_last ? __ldcg(part(c + i, mb) + u * (W4_BN / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < CU; ++i) {
              if (c + i > b_last) break;
#pragma unroll
              for (int u = 0; u < RU; ++u) {
                sum[u].x += v[i][u].x;
                sum[u].y += v[i][u].y;
                sum[u].z += v[i][u].z;
                sum[u].w += v[i][u].w;
              }
            }
          }
          if (n < p.N) {  // N is a multiple of 8
#pragma unroll
            for (int u = 0; u < RU; ++u)
              if (mb + u < rows) w4_store_out4<OUT_BF16, GATHER>(p, Cout, m0 + mb + u, n, sum[u]);
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ dequant
    // Set s (four warps, one per 32 rows = tensor-memory lanes 32 q .. 32 q + 31, the quadrant a warp may touch) converts
    // the slabs i with i % 2 == s into weight stage i % WS, which is free once the MMAs of slab i - WS have completed.
    // Whole slabs, because a hand-over costs a warp as much time as converting a quarter of one.
    const int sset = (warp - W4G_FIRST_DQ_WARP) >> 2;
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const uint32_t rawr = smem_u32(raw_base) + row * 128;
    const uint32_t sw = (uint32_t)(row & 7) << 4;  // 128-byte swizzle: quarter-warps read 8 rows x 8 distinct chunks
    const uint32_t st_addr = tmem_w + ((uint32_t)(q * 32) << 16);
    // ZT: this row's zero points of the slab's halves (128-wide groups: two rows)
    const uint32_t z_addr = smem_u32(z_base) + 2 * row;
    const uint32_t z_row1 = p.scale_rows == 2 ? 256u : 0u;
    const uint2 scalar_sub = make_uint2((0x6400u + (uint32_t)p.zero) * 0x00010001u, (0x5400u + ((uint32_t)p.zero << 4)) * 0x00010001u);
    const bool lead = lane == 0;
    // one loop per weight layout: a branch around the conversion inside it costs a register move per converted word
    auto convert_slabs = [&](auto il_) {
    uint32_t fail = 0;
    int ws = sset % WS;
#pragma unroll 1
    for (int i = sset; i < n_slabs; i += W4G_DQ_SETS) {
      const int rs = i % RS;
      const uint32_t rb = rawr + (uint32_t)rs * W4_RAW_PACKED;
      w4g_wait<W4G_RAW_FULL, ST_TIMEOUT_DEQUANT>(bar0 + 8 * rs, (uint32_t)(i / RS) & 1u, ctl, fail);
      uint4 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = w4g_lds128<0>(rb + ((uint32_t)(c << 4) ^ sw));
      uint2 sub[2] = {scalar_sub, scalar_sub};
      if constexpr (ZT) {
        uint16_t z0, z1;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(z0) : "r"(z_addr + rs * W4G_SC_BYTES));
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(z1) : "r"(z_addr + rs * W4G_SC_BYTES + z_row1));
        sub[0] = w4g_zero_subs((uint32_t)z0 * 0x00010001u);
        sub[1] = w4g_zero_subs((uint32_t)z1 * 0x00010001u);
      }
      const uint32_t bp = bar0 + 8 * ((i - WS) % W4G_BARS), ppar = (uint32_t)((i - WS) / W4G_BARS) & 1u;
      if (i >= WS) {
        if constexpr (Cfg::HALVES) w4g_wait<W4G_DONE0, ST_TIMEOUT_DEQUANT>(bp, ppar, ctl, fail);
        else w4g_wait<W4G_DONE, ST_TIMEOUT_DEQUANT>(bp, ppar, ctl, fail);
      }
      tc_fence_after_sync();
      const uint32_t ta = st_addr + ws * W4G_SLAB_COLS;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        if (Cfg::HALVES && c == 4) {
          tmem_st_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lead) w4g_arrive<W4G_W_FULL0>(bar0 + 8 * (i % W4G_BARS));
          if (i >= WS) w4g_wait<W4G_DONE, ST_TIMEOUT_DEQUANT>(bp, ppar, ctl, fail);
          tc_fence_after_sync();
        }
        uint32_t o[16];
        w4g_convert<decltype(il_)::value>(v[c], sub[c >> 2].x, sub[c >> 2].y, o);
        tmem_st_32x32b_x16(ta + 16 * c, o);
      }
      // the loads have delivered: hand the raw stage back
      __syncwarp();
      if (lead) w4g_arrive<W4G_RAW_EMPTY>(bar0 + 8 * rs);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lead) w4g_arrive<W4G_W_FULL>(bar0 + 8 * (i % W4G_BARS));
      ws += W4G_DQ_SETS;
      if (ws >= WS) ws -= WS;
      if ((i & 6) == 6) {
        fail = __any_sync(0xffffffffu, fail != 0) ? 1u : 0u;
        if (fail) break;
      }
    }
    };
    if (p.w_interleaved == 0) convert_slabs(std::integral_constant<bool, false>{});
    else convert_slabs(std::integral_constant<bool, true>{});
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (SMALL) cluster_sync_all();  // no CTA of the cluster leaves while another may still reach into it
  if (warp == W4G_FIRST_MMA_WARP + 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    if (lane == 0 && ctl_words[0] != 0 && p.status != nullptr) atomicMax(p.status, ctl_words[0]);
  }
}

}  // namespace qg
