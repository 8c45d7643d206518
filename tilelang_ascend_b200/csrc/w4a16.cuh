// W4A16 dequantize-GEMM for sm_100a, scale groups of 32 / 64 at up to 16 tokens (w4_route in qgemm_api.cu), and what the
// other W4A16 kernels share with it:
//   C[m, n] = cast( sum_k float(A[m, k]) * float(W[n, k]) ),  W[n, k] = half(q[n, k] - zero) * s[k / g, n]
// with q packed two per byte along K, low nibble first, in B_packed[N, K/2].
//
// The weight rows are the MMA "M" dimension (128 per tile, one TMEM lane per weight row) and the
// tokens are the MMA "N" dimension (MT = 16 per tile), so the memory-bound decode shapes stream
// the packed weights once at full tile height whatever the token count is.
//
// The dequantised weights never touch shared memory: each dequant thread owns one weight row, turns
// 32 bytes of nibbles into 64 f16 values in registers and writes them with tcgen05.st into a ring of
// tensor-memory columns, from which tcgen05.mma takes its A operand.  Shared memory only holds the
// packed weights and the (small) activation tiles.
//
// Persistent stream-K kernel: the (tile, 256-wide K slab) items are split evenly over the CTAs; a CTA
// whose slab range covers only part of a tile writes an fp32 partial into scratch memory, and the last
// contributor of that tile (found with a counter, never by waiting) adds the partials in a fixed order,
// so results do not depend on arrival order.
//   warp 0       TMA: packed weights [128 rows x 128 B] + the slab's scales into the "raw" ring
//   warp 1, 23..25  tcgen05.mma kind::f16 issuers (A from TMEM, B from shared memory), one fp32 accumulator
//                each in tensor memory, double buffered
//   warp 2       TMA: activation tiles [MT x 256 k] into their own ring
//   warps 3..6   epilogue (TMEM -> registers -> global / scratch, split-K reduction)
//   warps 7..22  dequant: lop3 magic-number conversion, (q - zero) * s in f16x2, tcgen05.st
// The conversion emits each group of eight K values in the order 0,4,1,5,2,6,3,7 (what the lop3 pairing
// gives for free).  A small pre-pass kernel (w4a16_prepare_activations) writes the activations once, in
// f16 and in that same K order, to scratch memory; the GEMM kernel loads them from there by TMA.
#pragma once

#include "common.cuh"

namespace qg {

struct W4A16Params {
  void* C;               // [M, N] f16 / bf16
  float* ws_partials;    // scratch: 2 * grid slots of [MT][128] fp32
  uint32_t* ws_counters; // scratch: grid counters, zeroed by the pre-pass kernel of every call
  int M, N, K;
  int group;            // quantisation group size along K
  int zero;             // integer zero point (0..15)
  int has_scales;       // 0: weights are the raw nibble values (scale 1)
  int batch;            // independent problems of the same shape (A, B_packed, scales, C all carry a leading batch dimension)
  int m_tiles, n_tiles, num_tiles;  // num_tiles = batch * n_tiles * m_tiles; tile = (b * n_tiles + n_tile) * m_tiles + m_tile
  int KS;               // 256-wide K slabs per tile
  // Group-sum kernel only: tiles 0 .. sk_tiles - 1 are cut stream-K fashion over all CTAs, then CTA c takes dp_rounds
  // whole tiles sk_tiles + c + j * grid.  The other kernels deal all (tile, slab) items evenly (total_items).
  int sk_tiles, dp_rounds;
  int sk_grid;  // wide tiles only: the first sk_tiles tiles are cut over this many CTAs
  // Group-sum kernel: in its single-launch form (no pre-pass) the caller's activations [batch, M, K], and whether they are
  // bf16; and whether the weight layout is the interleaved one.
  const void* A_raw;
  int a_is_bf16, w_interleaved;
  int scale_rows;       // scale rows fetched per slab (256 / group, at least 1)
  long long total_items;
  uint32_t* status;
  unsigned long long wait_limit_ns;
  int withhold;          // test hook of the two-CTA wide tiles (qgemm_debug_withhold_commit)
  // Gathered form (column-sharded weights, one process per GPU): when n_dst > 0 the [M, N] result is written
  // into columns [col0, col0 + N) of n_dst row-major [M, ldc] buffers, one per rank (this rank's own and its
  // peers', mapped into this process), instead of into C.  Plain stores to peer memory: the transfer of the
  // output overlaps the rest of the GEMM tile by tile, and no collective has to move it afterwards.
  void* c_dst[8];
  int n_dst, ldc, col0;
};

constexpr int W4_BN = 128;        // weight rows per tile
constexpr int W4_SLAB_K = 256;    // K per pipeline item: 128 packed bytes per row
constexpr int W4_DQ_WARPS = 16;
constexpr int W4_FIRST_DQ_WARP = 7;
constexpr int W4_MAX_MMA_WARPS = 4;
constexpr int W4_FIRST_XMMA_WARP = W4_FIRST_DQ_WARP + W4_DQ_WARPS;          // extra MMA-issuing warps 23..25
constexpr int W4_THREADS = (W4_FIRST_XMMA_WARP + W4_MAX_MMA_WARPS - 1) * 32;  // 832
constexpr int W4_RAW_PACKED = W4_BN * 128;         // 16 KB
constexpr int W4_RAW_BYTES = W4_RAW_PACKED + 2048; // + up to 8 scale rows of 128 halves
constexpr int W4_W_COLS = W4_SLAB_K / 2;           // TMEM columns per slab of dequantised weights

template <int MT>
struct W4Cfg {
  // Ring depths: a slot of the activation ring is recycled only after its item's MMAs have completed,
  // so that ring must cover the load latency plus the dequant and MMA time of the items in between.
  static_assert(MT == 16, "token tile");
  static constexpr int RAW_STAGES = 8;
  static constexpr int A_STAGES = 9;
  // One warp can issue a tcgen05.mma only every ~49 cycles (measured), far longer than a 16-token MMA runs,
  // so MMAW warps issue the K steps of a slab in parallel, each into its own accumulator; the epilogue adds
  // the MMAW accumulators in a fixed order.
  static constexpr int MMAW = 4;
  // Two accumulator sets: the epilogue of a segment overlaps the next segment's MMAs.
  static constexpr int ACC_BUFS = 2;
  static constexpr int W_STAGES = 3;
  static constexpr int A_KB_BYTES = MT * 128;          // one 64-wide K block of activations
  static constexpr int A_BYTES = 4 * A_KB_BYTES;       // one 256-wide slab
  static constexpr int ACC_COLS = ACC_BUFS * MMAW * MT;  // ACC_BUFS sets of MMAW accumulators
  static constexpr int TMEM_COLS = 512;
  static constexpr int BAR_BYTES = 512;
  static constexpr int SMEM_BYTES = RAW_STAGES * W4_RAW_BYTES + A_STAGES * A_BYTES + BAR_BYTES + 1024;
  static constexpr int CH = 16;  // accumulator columns per TMEM load
  static_assert(ACC_COLS + W_STAGES * W4_W_COLS <= 512, "tensor memory budget");
};

// Contiguous item range of CTA `b` out of `G`: [T*b/G, T*(b+1)/G).
__device__ __forceinline__ long long w4_range_begin(long long T, int G, int b) { return T * b / G; }
// The CTA whose range holds item i.
__device__ __forceinline__ int w4_owner(long long T, int G, long long i) { return (int)(((i + 1) * G - 1) / T); }

// tile -> batch index, first weight row, first token
template <int BN = W4_BN>
__device__ __forceinline__ void w4_tile_coords(const W4A16Params& p, int tile, int mt, int& b, int& n0, int& m0) {
  const int per_batch = p.n_tiles * p.m_tiles;
  b = tile / per_batch;
  const int t = tile - b * per_batch;
  n0 = (t / p.m_tiles) * BN;
  m0 = (t % p.m_tiles) * mt;
}

// One output value C[b][m][n] or, in the gathered form, column col0 + n of row m of every destination.
template <bool OUT_BF16, bool GATHER = true>
__device__ __forceinline__ void w4_store_out(const W4A16Params& p, uint16_t* Cout, int m, int n, float v) {
  const uint16_t h = OUT_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
  if (!GATHER || p.n_dst == 0) {
    Cout[(size_t)m * p.N + n] = h;
  } else {
    const size_t off = (size_t)m * p.ldc + p.col0 + n;
    // constant indices only: a run-time index into the kernel's parameter block would move it to local memory
#pragma unroll
    for (int d = 0; d < 8; ++d)
      if (d < p.n_dst) reinterpret_cast<uint16_t*>(p.c_dst[d])[off] = h;
  }
}

// Four consecutive output features n .. n + 3 of token m (N, ldc and col0 are multiples of 8): one 8-byte store each.
template <bool OUT_BF16, bool GATHER = true>
__device__ __forceinline__ void w4_store_out4(const W4A16Params& p, uint16_t* Cout, int m, int n, const float4& v) {
  const uint2 h = make_uint2(pack_out2<OUT_BF16>(v.x, v.y), pack_out2<OUT_BF16>(v.z, v.w));
  if (!GATHER || p.n_dst == 0) {
    *reinterpret_cast<uint2*>(Cout + (size_t)m * p.N + n) = h;
  } else {
    const size_t off = (size_t)m * p.ldc + p.col0 + n;
#pragma unroll
    for (int d = 0; d < 8; ++d)
      if (d < p.n_dst) *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.c_dst[d]) + off) = h;
  }
}

struct W4SegIter {
  long long item, end;
  int KS;
  __device__ __forceinline__ bool next(int& tile, int& ks0, int& ks1) {
    if (item >= end) return false;
    tile = (int)(item / KS);
    ks0 = (int)(item - (long long)tile * KS);
    const long long rem = end - item;
    ks1 = (rem < (long long)(KS - ks0)) ? (int)(ks0 + rem) : KS;
    item += ks1 - ks0;
    return true;
  }
};

// Eight packed nibbles n0..n7 (n_j at bits 4j) -> eight f16 values (n_j - zero) [* s], emitted as the
// half2 words (n0,n4) (n1,n5) (n2,n6) (n3,n7): the cheapest order for the magic-number conversion.
// Low nibbles: 0x6400 | n = 1024 + n, minus (1024 + zero).  High nibbles: 0x6400 | (n << 4) = 1024 + 16 n,
// times 1/16 minus (64 + zero).  Both are exact; the product with s rounds once (RN), like an f16 multiply.
__device__ __forceinline__ void w4_dequant8(uint32_t x, uint32_t sub_lo, uint32_t sub_hi, uint32_t s2, bool scaled,
                                            uint32_t* o) {
  uint32_t lo0, hi0, lo1, hi1;
  const uint32_t y = x >> 8;
  asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(lo0) : "r"(x));
  asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xea;" : "=r"(hi0) : "r"(x));
  asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;" : "=r"(lo1) : "r"(y));
  asm("lop3.b32 %0, %1, 0x00f000f0, 0x64006400, 0xea;" : "=r"(hi1) : "r"(y));
  const uint32_t sixteenth = 0x2C002C00u;  // 1/16
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(o[0]) : "r"(lo0), "r"(sub_lo));
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(o[1]) : "r"(hi0), "r"(sixteenth), "r"(sub_hi));
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(o[2]) : "r"(lo1), "r"(sub_lo));
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(o[3]) : "r"(hi1), "r"(sixteenth), "r"(sub_hi));
  if (scaled) {
    asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(o[0]) : "r"(s2));
    asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(o[1]) : "r"(s2));
    asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(o[2]) : "r"(s2));
    asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(o[3]) : "r"(s2));
  }
}

// Two raw nibble values -> weights under a zero point z2 and scale s2 (each twice), zero_mode 0 / 2: (q - z) * s, two
// roundings as the reference's sub.f16x2 + fma (tilelang/quantize/lop3.py:135-175, 325-358); 1: q * s - |z|, one.
__device__ __forceinline__ void w4_apply_zero(uint32_t& o, uint32_t s2, uint32_t z2, int zero_mode) {
  if (zero_mode == 1) {
    const uint32_t nz = z2 | 0x80008000u;  // -|z|, as the reference forms it (lop3.py:247)
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(o) : "r"(o), "r"(s2), "r"(nz));
  } else {
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(o) : "r"(o), "r"(z2));
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(o) : "r"(o), "r"(s2));
  }
}

__device__ __forceinline__ uint32_t w4_bf16x2_to_f16x2(uint32_t w) {
  const float lo = __uint_as_float(w << 16);
  const float hi = __uint_as_float(w & 0xffff0000u);
  return pack_f16x2(lo, hi);
}

// Eight consecutive K elements (a0..a7, as four 32-bit words) -> the words (a0,a4) (a1,a5) (a2,a6) (a3,a7).
__device__ __forceinline__ uint4 w4_permute_act(uint4 v) {
  uint4 o;
  o.x = __byte_perm(v.x, v.z, 0x5410);
  o.y = __byte_perm(v.x, v.z, 0x7632);
  o.z = __byte_perm(v.y, v.w, 0x5410);
  o.w = __byte_perm(v.y, v.w, 0x7632);
  return o;
}

// Pre-pass: activations [M, K] (f16 or bf16) -> f16 with every group of eight K values reordered to
// 0,4,1,5,2,6,3,7.  One 16-byte chunk per thread.  Block 0 also zeroes the split-K arrival counters, so
// every call starts from clean counters whatever an earlier (possibly aborted) call left in the scratch.
__global__ void __launch_bounds__(256)
w4a16_prepare_activations(const uint4* __restrict__ in, uint4* __restrict__ out, long long n_chunks, int is_bf16,
                          int permute, uint32_t* __restrict__ counters, int n_counters) {
  pdl_launch_dependents();  // the GEMM kernel behind may set up and start streaming weights meanwhile
  pdl_wait();               // the kernel in front (another call's GEMM, which lets its dependents start early) is done
  if (blockIdx.x == 0)
    for (int c = threadIdx.x; c < n_counters; c += blockDim.x) counters[c] = 0u;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_chunks) return;
  uint4 v = ld_written(in + i);
  if (is_bf16) {
    v.x = w4_bf16x2_to_f16x2(v.x);
    v.y = w4_bf16x2_to_f16x2(v.y);
    v.z = w4_bf16x2_to_f16x2(v.z);
    v.w = w4_bf16x2_to_f16x2(v.w);
  }
  // interleaved weights (every 32-bit word holding elements 0,2,4,6 | 1,3,5,7) decode in natural order
  out[i] = permute ? w4_permute_act(v) : v;
}

__device__ __forceinline__ void w4_epi_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

template <int MT, bool OUT_BF16>
__global__ void __launch_bounds__(W4_THREADS, 1)
w4a16_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS,
                  const __grid_constant__ CUtensorMap tmA, const W4A16Params p) {
  using Cfg = W4Cfg<MT>;
  pdl_launch_dependents();  // the next call's pre-pass may become resident; it waits for this grid before it writes
  constexpr int RS = Cfg::RAW_STAGES;
  constexpr int AS = Cfg::A_STAGES;
  constexpr int WS = Cfg::W_STAGES;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw_base = smem;
  uint8_t* a_base = smem + RS * W4_RAW_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(a_base + AS * Cfg::A_BYTES);
  uint64_t* raw_full = bars;
  uint64_t* raw_empty = raw_full + RS;
  uint64_t* a_full = raw_empty + RS;
  uint64_t* a_empty = a_full + AS;
  uint64_t* w_full = a_empty + AS;
  uint64_t* w_empty = w_full + WS;
  uint64_t* tfull = w_empty + WS;
  uint64_t* tempty = tfull + 2;
  uint64_t* drain = tempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* epi_flag = tmem_slot + 2;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RS; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], W4_DQ_WARPS);
    }
    for (int s = 0; s < AS; ++s) {
      mbar_init(&a_full[s], 1);
      // released by the one issuer that took the slab (round robin) or by all of them (K split)
      mbar_init(&a_empty[s], ((WS % Cfg::MMAW) == 0 && (AS % Cfg::MMAW) == 0) ? 1 : Cfg::MMAW);
    }
    for (int s = 0; s < WS; ++s) {
      mbar_init(&w_full[s], W4_DQ_WARPS);
      mbar_init(&w_empty[s], ((WS % Cfg::MMAW) == 0 && (AS % Cfg::MMAW) == 0) ? 1 : Cfg::MMAW);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], Cfg::MMAW);
      mbar_init(&tempty[i], 4);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    epi_flag[0] = epi_flag[1] = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
    if (p.has_scales) tma_prefetch_desc(&tmS);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_w = tmem_base + Cfg::ACC_COLS;  // ring of dequantised-weight columns
  const WaitCtl ctl{abort_flag, p.status, p.wait_limit_ns, 0};

  const int G = gridDim.x;
  const int cta = blockIdx.x;
  const long long T = p.total_items;
  W4SegIter seg{w4_range_begin(T, G, cta), w4_range_begin(T, G, cta + 1), p.KS};
  int tile, ks0, ks1;

  if (warp == 0) {
    // ------------------------------------------- raw producer: packed weights + scales
    if (lane == 0) {
      int rs = 0;
      uint32_t phase = 0, issued_mask = 0, parity_mask = 0;
      bool ok = true;
      const uint64_t once = l2_policy_evict_first();
      const uint32_t tx = W4_RAW_PACKED + (p.has_scales ? p.scale_rows * 256 : 0);
      while (ok && seg.next(tile, ks0, ks1)) {
        int b, n0, m0;
        w4_tile_coords(p, tile, MT, b, n0, m0);
        for (int ks = ks0; ks < ks1; ++ks) {
          if (!mbar_wait(&raw_empty[rs], phase ^ 1u, ctl, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
          uint8_t* dst = raw_base + rs * W4_RAW_BYTES;
          mbar_arrive_expect_tx(&raw_full[rs], tx);
          tma_load_3d_hint(dst, &tmW, &raw_full[rs], ks * (W4_SLAB_K / 2), n0, b, once);
          if (p.has_scales) {
            const int srow = (p.group <= W4_SLAB_K) ? ks * p.scale_rows : (ks * W4_SLAB_K) / p.group;
            tma_load_3d(dst + W4_RAW_PACKED, &tmS, &raw_full[rs], n0, srow, b);
          }
          issued_mask |= 1u << rs;
          parity_mask = (parity_mask & ~(1u << rs)) | (phase << rs);
          if (++rs == RS) { rs = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        for (int s = 0; s < RS; ++s) {
          if (!(issued_mask & (1u << s))) continue;
          const uint64_t t0 = global_timer_ns();
          while (!mbar_try_wait(&raw_full[s], (parity_mask >> s) & 1u)) {
            if (global_timer_ns() - t0 > p.wait_limit_ns) {
              if (p.status) atomicMax(p.status, (uint32_t)ST_TIMEOUT_DRAIN);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------- activation producer
    if (lane == 0) {
      pdl_wait();  // the prepared activations come from the pre-pass kernel in front of this one
      int as = 0;
      uint32_t phase = 0, issued_mask = 0, parity_mask = 0;
      bool ok = true;
      while (ok && seg.next(tile, ks0, ks1)) {
        int b, n0, m0;
        w4_tile_coords(p, tile, MT, b, n0, m0);
        for (int ks = ks0; ks < ks1; ++ks) {
          if (!mbar_wait(&a_empty[as], phase ^ 1u, ctl, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
          uint8_t* dstA = a_base + as * Cfg::A_BYTES;
          mbar_arrive_expect_tx(&a_full[as], Cfg::A_BYTES);
#pragma unroll
          for (int kb = 0; kb < 4; ++kb)
            tma_load_3d(dstA + kb * Cfg::A_KB_BYTES, &tmA, &a_full[as], ks * W4_SLAB_K + kb * 64, m0, b);
          issued_mask |= 1u << as;
          parity_mask = (parity_mask & ~(1u << as)) | (phase << as);
          if (++as == AS) { as = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        for (int s = 0; s < AS; ++s) {
          if (!(issued_mask & (1u << s))) continue;
          const uint64_t t0 = global_timer_ns();
          while (!mbar_try_wait(&a_full[s], (parity_mask >> s) & 1u)) {
            if (global_timer_ns() - t0 > p.wait_limit_ns) {
              if (p.status) atomicMax(p.status, (uint32_t)ST_TIMEOUT_DRAIN);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 1 || warp >= W4_FIRST_XMMA_WARP) {
    // -------------------------------------------------------------- MMA issuers
    // Each issuer accumulates into its own accumulator (columns w*MT of the buffer).  One issuing thread needs
    // 900-1400 cycles per slab for its MMAs, the commits and the barrier round trips, more than the slab's HBM
    // time, so the work is spread over MMAW threads, in one of two ways:
    //  - round robin (ring depths that are multiples of MMAW, so that an issuer always meets the same stages
    //    and every one of their phases, which its parity waits need): issuer w takes slab index % MMAW == w,
    //    all of its K steps;
    //  - K split (the 16- and 32-token tiles, whose rings are 3 / 9 and 2 / 6 deep): issuer w takes the K steps
    //    kk = w, w + MMAW, ... of every slab.  Following every slab just to keep the parity waits safe made
    //    round robin no faster there (measured), and those tiles are bound by the dequant warps anyway.
    const int mw = (warp == 1) ? 0 : (warp - W4_FIRST_XMMA_WARP + 1);
    // The issuing warps run converged: all lanes wait, one hardware-elected lane (always the same one) issues.  Under
    // `if (elect_one_sync())` the compiler knows a single lane runs and keeps descriptors in uniform registers.  Issue
    // time is what matters here: one thread needs 100-130 cycles per tcgen05.mma with the dequant warps competing for
    // issue slots, i.e. ~2000 cycles for a slab's 16 MMAs, which themselves run for 1024 (ablations at 512 tokens,
    // N=28672: 284 us; 173 us without the MMAs; 232 us without the conversion arithmetic).  The elected lane took
    // that case from 284 to 228 us.
    if (mw < Cfg::MMAW) {
      constexpr uint32_t idesc = make_idesc(ACC_F32, FMT_F16, FMT_F16, 0, 0, W4_BN, MT);
      const uint64_t desc_hi = make_desc_kmajor(0);  // K-major activation descriptor without its start address
      const uint32_t a_base_u32 = smem_u32(a_base);
      int ws = 0, as = 0;
      uint32_t wphase = 0, aphase = 0;
      // With ring depths that are multiples of MMAW an issuer always meets the same stages and every one of
      // their phases; otherwise it has to follow the other issuers' slabs too (see below).
      constexpr bool ROUND_ROBIN = (WS % Cfg::MMAW) == 0 && (AS % Cfg::MMAW) == 0;
      int it = 0;
      int turn = 0;  // slab index % MMAW
      bool ok = true;
      while (ok && seg.next(tile, ks0, ks1)) {
        const int buf = it % Cfg::ACC_BUFS;
        const uint32_t tphase = (uint32_t)(it / Cfg::ACC_BUFS) & 1u;
        if (!mbar_wait_warp(&tempty[buf], tphase ^ 1u, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after_sync();
        const uint32_t d = tmem_base + buf * (Cfg::MMAW * MT) + mw * MT;
        uint32_t started = 0;  // 0 for this issuer's first MMA of the segment: overwrite the accumulator
        for (int ks = ks0; ks < ks1; ++ks) {
          if (!ROUND_ROBIN || turn == mw) {
            if (!mbar_wait_warp(&a_full[as], aphase, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
            if (!mbar_wait_warp(&w_full[ws], wphase, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
            tc_fence_after_sync();
            const uint64_t adesc0 = desc_hi | (uint64_t)(((a_base_u32 + as * Cfg::A_BYTES) & 0x3FFFFu) >> 4);
            const uint32_t tW = tmem_w + ws * W4_W_COLS;
            constexpr int STEPS = ROUND_ROBIN ? W4_SLAB_K / 16 : (W4_SLAB_K / 16) / Cfg::MMAW;
            if (elect_one_sync()) {
#pragma unroll
              for (int j = 0; j < STEPS; ++j) {  // 16 k per MMA: 8 TMEM columns, 32 bytes of smem
                const int kk = ROUND_ROBIN ? j : j * Cfg::MMAW + mw;
                const uint32_t off = (uint32_t)(((kk >> 2) * Cfg::A_KB_BYTES + (kk & 3) * 32) >> 4);
                umma_f16_ts(d, tW + kk * 8, adesc0 + off, idesc, j == 0 ? started : 1u);
              }
              umma_commit(&w_empty[ws]);
              umma_commit(&a_empty[as]);
            }
            started = 1u;
          }
          if (++turn == Cfg::MMAW) turn = 0;
          if (++ws == WS) { ws = 0; wphase ^= 1u; }
          if (++as == AS) { as = 0; aphase ^= 1u; }
        }
        // the elected lane is the same one every time, so this commit covers the MMAs issued above
        if (ok && elect_one_sync()) umma_commit(&tfull[buf]);
        ++it;
      }
      if (!ok && mw == 0) {
        if (elect_one_sync()) umma_commit(drain);
        if (lane == 0) {
          const uint64_t t0 = global_timer_ns();
          while (!mbar_try_wait(drain, 0)) {
            if (global_timer_ns() - t0 > p.wait_limit_ns) break;
          }
        }
      }
    }
  } else if (warp >= 3 && warp < W4_FIRST_DQ_WARP) {
    // ---------------------------------------------------------------- epilogue
    constexpr int CH = Cfg::CH;
    const int q = warp & 3;
    const int nl = q * 32 + lane;  // weight row inside the tile == TMEM lane
    pdl_wait();  // the arrival counters are zeroed by the pre-pass kernel in front of this one
    int it = 0, seg_idx = 0;
    constexpr bool ROUND_ROBIN_E = (WS % Cfg::MMAW) == 0 && (AS % Cfg::MMAW) == 0;  // as in the MMA issuers
    long long first_slab = 0;  // CTA-local index of the segment's first slab: issuer (first_slab + i) % MMAW took slab i
    while (seg.next(tile, ks0, ks1)) {
      const int buf = it % Cfg::ACC_BUFS;
      const uint32_t tphase = (uint32_t)(it / Cfg::ACC_BUFS) & 1u;
      ++it;
      const int seg_len = ks1 - ks0;
      const int first_turn = (int)(first_slab % Cfg::MMAW);
      first_slab += seg_len;
      int b, n0, m0;
      w4_tile_coords(p, tile, MT, b, n0, m0);
      const int n = n0 + nl;
      uint16_t* Cout = reinterpret_cast<uint16_t*>(p.C) + (size_t)b * p.M * p.N;
      const bool full_tile = (ks0 == 0 && ks1 == p.KS);
      const int my_slot = (ks1 < p.KS) ? 2 * cta + 1 : 2 * cta;
      const bool ok = mbar_wait_warp(&tfull[buf], tphase, ctl, ST_TIMEOUT_EPILOGUE);
      if (ok) {
        tc_fence_after_sync();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * (Cfg::MMAW * MT);
#pragma unroll 1
        for (int c = 0; c < MT / CH; ++c) {
          uint32_t r[CH];
#pragma unroll
          for (int j = 0; j < CH; ++j) r[j] = 0u;  // +0.0f
#pragma unroll
          for (int a = 0; a < Cfg::MMAW; ++a) {  // add the issuers' accumulators in fixed order
            // issuer a wrote its accumulator in this segment only if one of the segment's slabs was its turn
            if (!ROUND_ROBIN_E || ((a - first_turn + Cfg::MMAW) % Cfg::MMAW) < seg_len) {
              uint32_t r2[CH];
              tmem_ld_32x32b_x16(taddr + a * MT + c * CH, r2);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < CH; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(r2[j]));
            }
          }
          if (full_tile) {
            if (n < p.N) {
#pragma unroll
              for (int j = 0; j < CH; ++j) {
                const int m = m0 + c * CH + j;
                if (m < p.M) {
                  const float v = __uint_as_float(r[j]);
                  w4_store_out<OUT_BF16>(p, Cout, m, n, v);
                }
              }
            }
          } else {
            float* dst = p.ws_partials + (size_t)my_slot * (MT * W4_BN) + (size_t)(c * CH) * W4_BN + nl;
#pragma unroll
            for (int j = 0; j < CH; ++j) dst[j * W4_BN] = __uint_as_float(r[j]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[buf]);
      }
      // Segment end.  The four epilogue warps decide together whether to go on (a warp that left alone would
      // leave the others waiting at the named barrier for ever): a wait that gave up set the abort flag before its
      // warp reached the barrier below; one thread reads the flag once and publishes it, with the split-K
      // outcome, in a control word that alternates between two slots by segment, so that a fast warp's next
      // write cannot overtake a slow warp's read.
      const int par = seg_idx & 1;
      ++seg_idx;
      const long long first_item = (long long)tile * p.KS;
      int b_first = 0, b_last = 0;
      if (!full_tile) {
        b_first = w4_owner(T, G, first_item);
        b_last = w4_owner(T, G, first_item + p.KS - 1);
        __threadfence();
      }
      w4_epi_bar();
      if (warp == 3 && lane == 0) {
        uint32_t ctrl = *abort_flag ? 1u : 0u;
        if (!ctrl && !full_tile) {
          // split tile: count arrivals; the last contributor reduces in a fixed order
          const uint32_t old = atomicAdd(p.ws_counters + b_first, 1u);
          if (old == (uint32_t)(b_last - b_first)) ctrl |= 2u;
        }
        epi_flag[par] = ctrl;
      }
      w4_epi_bar();
      const uint32_t ctrl = epi_flag[par];
      if (ctrl & 1u) break;
      const bool is_last = (ctrl & 2u) != 0;
      if (is_last) {
        __threadfence();
        if (n < p.N) {
          // Fixed summation order (contributor b_first .. b_last); per contributor all MT loads are issued
          // before the first add so that their latencies overlap.
          constexpr int RU = 16;
          const int rows = min(MT, p.M - m0);
#pragma unroll 1
          for (int mb = 0; mb < rows; mb += RU) {
            float sum[RU];
#pragma unroll
            for (int u = 0; u < RU; ++u) sum[u] = 0.0f;
#pragma unroll 1
            for (int c = b_first; c <= b_last; ++c) {
              const long long c_end = w4_range_begin(T, G, c + 1);
              const int slot = (c_end >= first_item + p.KS) ? 2 * c : 2 * c + 1;
              const float* src = p.ws_partials + (size_t)slot * (MT * W4_BN) + (size_t)mb * W4_BN + nl;
              float v[RU];
#pragma unroll
              for (int u = 0; u < RU; ++u) v[u] = (mb + u < rows) ? __ldcg(src + u * W4_BN) : 0.0f;
#pragma unroll
              for (int u = 0; u < RU; ++u) sum[u] += v[u];
            }
#pragma unroll
            for (int u = 0; u < RU; ++u) {
              if (mb + u < rows)
                w4_store_out<OUT_BF16>(p, Cout, m0 + mb + u, n, sum[u]);
            }
          }
        }
      }
    }
  } else if (warp >= W4_FIRST_DQ_WARP && warp < W4_FIRST_XMMA_WARP) {
    // ----------------------------------------------------------------- dequant
    // Warp (q, j): TMEM lanes 32q..32q+31 (the quadrant this warp may touch), K sub-range [64j, 64j+64) of
    // the slab = packed 16-byte chunks 2j and 2j+1 of the row = 32 TMEM columns.
    const int wd = warp - W4_FIRST_DQ_WARP;
    const int q = warp & 3;
    const int j = wd >> 2;
    const int row = q * 32 + lane;
    const int sw = row & 7;
    const uint32_t off0 = row * 128 + (((2 * j) ^ sw) << 4);      // quarter-warps read 8 rows x 8 distinct chunks
    const uint32_t off1 = row * 128 + (((2 * j + 1) ^ sw) << 4);
    const uint32_t zero = (uint32_t)p.zero;
    const uint32_t sub_lo = (0x6400u + zero) * 0x00010001u;                      // (1024 + zero) x2
    const uint32_t sub_hi = ((0x5400u + (zero << 4)) | 0x8000u) * 0x00010001u;   // -(64 + zero) x2
    const bool scaled = p.has_scales != 0;
    const int srow0 = (p.group <= W4_SLAB_K) ? (64 * j) / p.group : 0;
    const int srow1 = (p.group <= W4_SLAB_K) ? (64 * j + 32) / p.group : 0;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    int rs = 0, ws = 0;
    uint32_t rphase = 0, wphase = 0;
    bool ok = true;
    while (ok && seg.next(tile, ks0, ks1)) {
      for (int ks = ks0; ks < ks1; ++ks) {
        if (!mbar_wait_warp(&raw_full[rs], rphase, ctl, ST_TIMEOUT_DEQUANT)) { ok = false; break; }
        const uint8_t* rawp = raw_base + rs * W4_RAW_BYTES;
        const uint4 v0 = *reinterpret_cast<const uint4*>(rawp + off0);
        const uint4 v1 = *reinterpret_cast<const uint4*>(rawp + off1);
        uint32_t s20 = 0x3C003C00u, s21 = 0x3C003C00u;
        if (scaled) {
          const __half* sS = reinterpret_cast<const __half*>(rawp + W4_RAW_PACKED);
          s20 = (uint32_t)__half_as_ushort(sS[srow0 * W4_BN + row]) * 0x00010001u;
          s21 = (uint32_t)__half_as_ushort(sS[srow1 * W4_BN + row]) * 0x00010001u;
        }
        uint32_t o[32];
        w4_dequant8(v0.x, sub_lo, sub_hi, s20, scaled, o + 0);
        w4_dequant8(v0.y, sub_lo, sub_hi, s20, scaled, o + 4);
        w4_dequant8(v0.z, sub_lo, sub_hi, s20, scaled, o + 8);
        w4_dequant8(v0.w, sub_lo, sub_hi, s20, scaled, o + 12);
        w4_dequant8(v1.x, sub_lo, sub_hi, s21, scaled, o + 16);
        w4_dequant8(v1.y, sub_lo, sub_hi, s21, scaled, o + 20);
        w4_dequant8(v1.z, sub_lo, sub_hi, s21, scaled, o + 24);
        w4_dequant8(v1.w, sub_lo, sub_hi, s21, scaled, o + 28);
        // the packed bytes are in registers: hand the raw stage back to the producer
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[rs]);
        if (++rs == RS) { rs = 0; rphase ^= 1u; }

        if (!mbar_wait_warp(&w_empty[ws], wphase ^ 1u, ctl, ST_TIMEOUT_DEQUANT)) { ok = false; break; }
        tc_fence_after_sync();
        tmem_st_32x32b_x32(tmem_w + lane_addr + ws * W4_W_COLS + j * 32, o);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&w_full[ws]);
        if (++ws == WS) { ws = 0; wphase ^= 1u; }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

}  // namespace qg
