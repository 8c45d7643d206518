// W4A16 dequantize-GEMM, sm_100a, for more than 64 tokens (and what the kernels for fewer do not take): tiles of 128 weight
// rows x up to 256 tokens.
//   C[m, n] = cast( sum_k float(A[m, k]) * float(W[n, k]) ),  W[n, k] = half(q - zero) * s as in w4a16.cuh, bit for bit
//
// What bounds these shapes is the conversion of the packed weights and the tensor pipe, in that order: turning a 16 KB
// slab (128 rows x 256 k) into f16 costs an SM about 1700 cycles of issue slots whatever the tile's tokens, the slab's
// MMAs 8 cycles per token.  So a converted slab serves as many tokens as the accumulators have room for: 256 columns of
// tensor memory hold one accumulator of up to 256 tokens (or two of up to 128), the other 256 four stages of converted
// weights of 128 k each.  At 256 tokens the MMAs of a slab (2048 cycles) cover its conversion, which 128 tokens (1024
// cycles) do not.  The tokens are cut into tiles of equal height, a multiple of 16 (500 tokens: two tiles of 256; 300:
// two of 160), so hardly any work is spent on padding.
// Measured (K = 8192, N = 28672; before: 128-token tiles, from 1792 tokens on weights dequantised to memory once and
// an f16 GEMM): 128 tokens 79.5 -> 65 us, 256: 128 -> 97, 500: 234 -> 180, 1024: 447 -> 338, 4096: 1613 -> 1390 - 1550 us;
// a zeros tensor, 100 tokens: 249 -> 95 us.  Without the activation loads 500 tokens take 153 us, without the conversion's
// arithmetic 160, without the MMAs 107, with the MMAs alone 133: no single role sets the pace any more.
//
// Structure (persistent; tiles dealt as w4_wide_plan says: first the tiles cut along K, then whole ones), 28 warps:
//   warp 0        TMA: packed weights + scale (and zero) rows, one slab per stage
//   warp 1        TMA: prepared activations, [tile tokens x 64 k] per stage
//   warp 2        tcgen05.mma kind::f16 issuer (A = weights from tensor memory, B = activations from shared memory)
//   (two CTAs may share a tile of 256 weight rows, see PAIR)
//   warp 3        allocates tensor memory
//   warps 4..11   epilogue: two sets of four warps take 16 tokens in turn; the accumulator is handed back as soon as it
//                 has been read, the split-K sum runs beside the next tile's MMAs
//   warps 12..27  dequant: warp (q, j) rows 32 q .. + 31, k 64 j .. + 63 of every slab
#pragma once

#include "common.cuh"
#include "w4a16.cuh"
#include "w4a16_gs.cuh"

namespace qg {

constexpr int W4W_MAX_MT = 256;
// A tile's tokens are the MMA's N: a multiple of 16 for one CTA's 128 rows.  For the 256 rows of two CTAs multiples of 32 are
// taken, which every statement of the shape rules for cta_group::2 allows; some allow steps of 16 as well, some do not.
constexpr int W4W_MT_STEP = 16, W4W_PAIR_MT_STEP = 32;
static_assert(W4W_MAX_MT % W4W_PAIR_MT_STEP == 0, "tile heights");
constexpr int W4W_FIRST_EPI_WARP = 4;
constexpr int W4W_EPI_WARPS = 8;
constexpr int W4W_FIRST_DQ_WARP = W4W_FIRST_EPI_WARP + W4W_EPI_WARPS;  // 12
constexpr int W4W_DQ_WARPS = 16;
constexpr int W4W_THREADS = (W4W_FIRST_DQ_WARP + W4W_DQ_WARPS) * 32;   // 896
constexpr int W4W_RS = 3;                         // packed-weight ring, in slabs
constexpr int W4W_WS = 4;                         // converted-weight ring (tensor memory), in halves of a slab
constexpr int W4W_W_COLS = 64;                    // columns of a half
constexpr int W4W_ACC_COLS = 256;
constexpr int W4W_A_RING_BYTES = 160 * 1024;      // activations: as many stages of mt x 128 bytes as fit, at most:
constexpr int W4W_MAX_AS = 10;
constexpr int W4W_BAR_BYTES = 512;

template <bool ZT>
struct W4WideCfg {
  static constexpr int RAW_BYTES = W4_RAW_BYTES + (ZT ? 2048 : 0);  // packed rows, up to 8 scale rows, up to 8 zero rows
  static constexpr int SMEM_BYTES = W4W_A_RING_BYTES + W4W_RS * RAW_BYTES + W4W_BAR_BYTES + 1024;
  static_assert(SMEM_BYTES <= 232448, "shared memory of a CTA");
};

// 16-bit outputs of four tokens m .. m + 3 and this lane's output feature n (see transpose_tokens4; N, ldc and col0 are
// multiples of 8).
__device__ __forceinline__ void w4w_store_tokens4(const W4A16Params& p, uint16_t* Cout, int m, int n, int lane, uint32_t w01,
                                                  uint32_t w23) {
  int row = m, col = n;
  const uint2 v = transpose_tokens4(lane, w01, w23, row, col);
  if (row >= p.M || col >= p.N) return;
  if (p.n_dst == 0) {
    *reinterpret_cast<uint2*>(Cout + (size_t)row * p.N + col) = v;
  } else {
    const size_t off = (size_t)row * p.ldc + p.col0 + col;
#pragma unroll
    for (int d = 0; d < 8; ++d)
      if (d < p.n_dst) *reinterpret_cast<uint2*>(reinterpret_cast<uint16_t*>(p.c_dst[d]) + off) = v;
  }
}

// ZT: zero points from a [K/group, N] f16 tensor in any of the three modes (w4_apply_zero).
// PAIR: a cluster of two CTAs makes tiles of 256 weight rows with MMAs over both (tcgen05.mma.cta_group::2): each CTA converts its
// own 128 rows into its own tensor memory, holds their accumulators, and loads half of the tile's tokens, which the tensor cores
// of both read.  At 256 tokens one CTA by itself takes 36 KB from L2 per 64 k, whose MMAs last 512 cycles, more than the 64 bytes
// a cycle that reach an SM; a pair 20 KB each.  The leader (rank 0) issues; converted weights, activations and free accumulators
// of both CTAs are signalled on its barriers, its commits signal both.  Figures and the choice: w4_wide_plan in qgemm_api.cu.
template <bool OUT_BF16, bool ZT, bool PAIR>
__global__ void __launch_bounds__(W4W_THREADS, 1)
w4a16_wide_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS,
                  const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmA,
                  const __grid_constant__ W4A16Params p, const int mt, const int zero_mode) {
  using Cfg = W4WideCfg<ZT>;
  constexpr int RS = W4W_RS, WS = W4W_WS;
  pdl_launch_dependents();  // the next call's pre-pass may become resident; it waits for this grid before it writes

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a_base = smem;
  uint8_t* raw_base = smem + W4W_A_RING_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(raw_base + RS * Cfg::RAW_BYTES);
  uint64_t* raw_full = bars;
  uint64_t* raw_empty = raw_full + RS;
  uint64_t* a_full = raw_empty + RS;
  uint64_t* a_empty = a_full + W4W_MAX_AS;
  uint64_t* w_full = a_empty + W4W_MAX_AS;
  uint64_t* w_empty = w_full + WS;
  uint64_t* tfull = w_empty + WS;
  uint64_t* tempty = tfull + 2;
  uint64_t* drain = tempty + 2;
  uint64_t* reported = drain + 1;  // PAIR: the second CTA's producer of activations has ended (pair_wait_copies)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile uint32_t* epi_flag = tmem_slot + 2;  // two words
  uint32_t* peer_issued = tmem_slot + 4;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int crank = PAIR ? (int)cluster_ctarank() : 0;
  const int a_rows = PAIR ? mt / 2 : mt;                            // tokens that this CTA loads
  const int a_bytes = a_rows * 128;                                 // one stage: their 64 k
  const int AS = min(W4W_MAX_AS, W4W_A_RING_BYTES / a_bytes);
  const int acc_bufs = mt <= W4W_ACC_COLS / 2 ? 2 : 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < RS; ++s) {
      mbar_init(&raw_full[s], 1);
      mbar_init(&raw_empty[s], W4W_DQ_WARPS);
    }
    for (int s = 0; s < W4W_MAX_AS; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&a_empty[s], 1);
    }
    for (int s = 0; s < WS; ++s) {
      mbar_init(&w_full[s], (PAIR ? 2 : 1) * W4W_DQ_WARPS / 2);  // PAIR: both CTAs' warps, on the leader's barrier
      mbar_init(&w_empty[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], (PAIR ? 2 : 1) * W4W_EPI_WARPS);
    }
    mbar_init(drain, 1);
    mbar_init(reported, 1);
    *abort_flag = 0;
    epi_flag[0] = epi_flag[1] = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmA);
    if (p.has_scales) tma_prefetch_desc(&tmS);
    if (ZT) tma_prefetch_desc(&tmZ);
  }
  if (warp == 3) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if constexpr (PAIR) cluster_sync_all();  // both CTAs' barriers exist before either signals the other's
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tmem_w = tmem_base + W4W_ACC_COLS;
  const WaitCtl ctl{abort_flag, p.status, p.wait_limit_ns, 0};

  const int G = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;  // workers: CTAs, or pairs of them
  const int cta = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int n_off = crank * W4_BN;                              // PAIR: a tile is 256 weight rows, 128 for each CTA
  // where this CTA's partial sums and its tile's arrival counter are: each CTA of a pair has its own
  auto partial_slot = [&](int worker, int second) { return PAIR ? 2 * (2 * worker + second) + crank : 2 * worker + second; };
  auto counter = [&](int worker) { return p.ws_counters + (PAIR ? 2 * worker + crank : worker); };
  auto arrive_leader = [&](uint64_t* bar) {  // on the leader's barrier
    if constexpr (PAIR) mbar_arrive_leader(bar);
    else mbar_arrive(bar);
  };
  // the first sk_tiles tiles' slabs, dealt evenly to the first Gs CTAs as contiguous ranges
  const long long T = (long long)p.sk_tiles * p.KS;
  const int Gs = p.sk_grid;
  const long long item0 = cta < Gs ? w4_range_begin(T, Gs, cta) : T, item1 = cta < Gs ? w4_range_begin(T, Gs, cta + 1) : T;
  const int whole = (p.num_tiles - p.sk_tiles - cta + G - 1) / G;  // this worker's whole tiles
  W4HybridIter seg{W4SegIter{item0, item1, p.KS}, p.sk_tiles + cta, whole, G, p.KS};
  int tile, ks0, ks1;

  if (warp == 0 || warp == 1) {
    // ------------------------------------------------------------------ producers
    if (lane == 0) {
      int st = 0;
      uint32_t phase = 0, issued_mask = 0, parity_mask = 0, fills = 0;
      bool ok = true;
      if (warp == 0) {
        const uint32_t row_tx = (uint32_t)p.scale_rows * 256u;
        const uint32_t tx = W4_RAW_PACKED + (p.has_scales ? row_tx : 0u) + (ZT ? row_tx : 0u);
        while (ok && seg.next(tile, ks0, ks1)) {
          int b, n0, m0;
          w4_tile_coords<PAIR ? 2 * W4_BN : W4_BN>(p, tile, mt, b, n0, m0);
          for (int ks = ks0; ks < ks1; ++ks) {
            if (!mbar_wait(&raw_empty[st], phase ^ 1u, ctl, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
            uint8_t* dst = raw_base + st * Cfg::RAW_BYTES;
            mbar_arrive_expect_tx(&raw_full[st], tx);
            tma_load_3d(dst, &tmW, &raw_full[st], ks * (W4_SLAB_K / 2), n0 + n_off, b);
            const int srow = (p.group <= W4_SLAB_K) ? ks * p.scale_rows : (ks * W4_SLAB_K) / p.group;
            if (p.has_scales) tma_load_3d(dst + W4_RAW_PACKED, &tmS, &raw_full[st], n0 + n_off, srow, b);
            if (ZT) tma_load_3d(dst + W4_RAW_BYTES, &tmZ, &raw_full[st], n0 + n_off, srow, b);
            issued_mask |= 1u << st;
            parity_mask = (parity_mask & ~(1u << st)) | (phase << st);
            if (++st == RS) { st = 0; phase ^= 1u; }
          }
        }
      } else {
        pdl_wait();  // the prepared activations come from the pre-pass kernel in front of this one
        const bool idle = PAIR && p.withhold == 3 + crank && cta == G - 1;  // test hook: this CTA copies nothing
        while (!idle && ok && seg.next(tile, ks0, ks1)) {
          int b, n0, m0;
          w4_tile_coords<PAIR ? 2 * W4_BN : W4_BN>(p, tile, mt, b, n0, m0);
          for (int kb = 4 * ks0; kb < 4 * ks1; ++kb) {
            if (!mbar_wait(&a_empty[st], phase ^ 1u, ctl, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
            if constexpr (PAIR) {  // both CTAs' bytes are counted on the leader's barrier
              if (crank == 0) mbar_arrive_expect_tx(&a_full[st], 2u * (uint32_t)a_bytes);
              tma_load_3d_pair(a_base + st * a_bytes, &tmA, mapa_u32(smem_u32(&a_full[st]), 0), kb * 64, m0 + crank * a_rows, b);
            } else {
              mbar_arrive_expect_tx(&a_full[st], (uint32_t)a_bytes);
              tma_load_3d(a_base + st * a_bytes, &tmA, &a_full[st], kb * 64, m0, b);
            }
            ++fills;
            issued_mask |= 1u << st;
            parity_mask = (parity_mask & ~(1u << st)) | (phase << st);
            if (++st == AS) { st = 0; phase ^= 1u; }
          }
        }
      }
      if (PAIR && warp == 1) {
        pair_wait_copies(a_full, (uint32_t)AS, (uint32_t)a_bytes, fills, crank, reported, peer_issued, ctl);
      } else if (!ok) {  // wait (bounded) for the copies still in flight before the CTA may exit
        uint64_t* full = warp == 0 ? raw_full : a_full;
        for (int s = 0; s < W4W_MAX_AS; ++s) {
          if (!(issued_mask & (1u << s))) continue;
          const uint64_t t0 = global_timer_ns();
          while (!mbar_try_wait(&full[s], (parity_mask >> s) & 1u)) {
            if (global_timer_ns() - t0 > p.wait_limit_ns) {
              if (p.status) atomicMax(p.status, (uint32_t)ST_TIMEOUT_DRAIN);
              break;
            }
          }
        }
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ MMA issuer (converged warp, one elected lane)
    const uint32_t idesc = make_idesc(ACC_F32, FMT_F16, FMT_F16, 0, 0, PAIR ? 2 * W4_BN : W4_BN, mt);
    const uint64_t desc_hi = make_desc_kmajor(0);  // K-major activation descriptor without its start address
    const uint32_t a_base_u32 = smem_u32(a_base);
    auto commit = [](uint64_t* bar) {
      if constexpr (PAIR) umma_commit_pair(bar);
      else umma_commit(bar);
    };
    int as = 0, ws = 0, it = 0;
    uint32_t aphase = 0, wphase = 0;
    bool ok = true;
    while ((!PAIR || crank == 0) && ok && seg.next(tile, ks0, ks1)) {  // PAIR: the leader's, for both CTAs
      const int buf = acc_bufs == 2 ? it & 1 : 0;
      const uint32_t tphase = (uint32_t)(acc_bufs == 2 ? it >> 1 : it) & 1u;
      ++it;
      if (!mbar_wait_warp(&tempty[buf], tphase ^ 1u, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t d = tmem_base + buf * (W4W_ACC_COLS / 2);
      for (int h = 2 * ks0; ok && h < 2 * ks1; ++h) {
        if (!mbar_wait_warp(&w_full[ws], wphase, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
        const uint32_t tW = tmem_w + ws * W4W_W_COLS;
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          if (!mbar_wait_warp(&a_full[as], aphase, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
          tc_fence_after_sync();
          const uint64_t adesc = desc_hi | (uint64_t)(((a_base_u32 + as * a_bytes) & 0x3FFFFu) >> 4);
          if (elect_one_sync()) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {  // 16 k per MMA: 8 tensor-memory columns, 32 bytes of a row
              const uint32_t add = (h != 2 * ks0 || blk != 0 || kk != 0) ? 1u : 0u;
              if constexpr (PAIR) umma_f16_ts_pair(d, tW + blk * 32 + kk * 8, adesc + 2 * kk, idesc, add);
              else umma_f16_ts(d, tW + blk * 32 + kk * 8, adesc + 2 * kk, idesc, add);
            }
            commit(&a_empty[as]);
            if (blk == 1) commit(&w_empty[ws]);
          }
          if (++as == AS) { as = 0; aphase ^= 1u; }
        }
        if (++ws == WS) { ws = 0; wphase ^= 1u; }
      }
      const bool withheld = PAIR && p.withhold == 1 && cta == G - 1 && seg.done();
      if (ok && !withheld && elect_one_sync()) commit(&tfull[buf]);  // the elected lane is the same one every time
    }
    if (!ok) {
      if (elect_one_sync()) commit(drain);
      if (lane == 0) {
        const uint64_t t0 = global_timer_ns();
        while (!mbar_try_wait(drain, 0)) {
          if (global_timer_ns() - t0 > p.wait_limit_ns) break;
        }
      }
    }
  } else if (warp >= W4W_FIRST_EPI_WARP && warp < W4W_FIRST_DQ_WARP) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const int e = (warp - W4W_FIRST_EPI_WARP) >> 2;  // set e takes the 16-token pieces of parity e
    const int nl = q * 32 + lane;                    // weight row inside the tile == TMEM lane
    pdl_wait();  // the arrival counters are zeroed by the pre-pass kernel in front of this one
    int it = 0;
    while (seg.next(tile, ks0, ks1)) {
      const int buf = acc_bufs == 2 ? it & 1 : 0;
      const uint32_t tphase = (uint32_t)(acc_bufs == 2 ? it >> 1 : it) & 1u;
      int b, n0, m0;
      w4_tile_coords<PAIR ? 2 * W4_BN : W4_BN>(p, tile, mt, b, n0, m0);
      const int n = n0 + n_off + nl;
      uint16_t* Cout = reinterpret_cast<uint16_t*>(p.C) + (size_t)b * p.M * p.N;
      const bool full_tile = (ks0 == 0 && ks1 == p.KS);
      const int my_slot = partial_slot(cta, ks1 < p.KS ? 1 : 0);
      float* part = p.ws_partials + (size_t)my_slot * ((size_t)mt * W4_BN) + nl;
      if (mbar_wait_warp(&tfull[buf], tphase, ctl, ST_TIMEOUT_EPILOGUE)) {
        tc_fence_after_sync();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * (W4W_ACC_COLS / 2);
#pragma unroll 1
        for (int c = 16 * e; c < mt; c += 32) {
          uint32_t r[16];
          tmem_ld_32x32b_x16(taddr + c, r);
          tmem_ld_wait();
          if (full_tile) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              w4w_store_tokens4(p, Cout, m0 + c + j, n, lane,
                                pack_out2<OUT_BF16>(__uint_as_float(r[j]), __uint_as_float(r[j + 1])),
                                pack_out2<OUT_BF16>(__uint_as_float(r[j + 2]), __uint_as_float(r[j + 3])));
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) part[(c + j) * W4_BN] = __uint_as_float(r[j]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) arrive_leader(&tempty[buf]);
      }
      // Segment end.  The epilogue warps decide together whether to go on (a warp that left alone would leave the others
      // waiting at the named barrier for ever): a wait that gave up set the abort flag before its warp reached the first
      // barrier; one thread reads the flag once and publishes it, with the split-K outcome, in a control word that
      // alternates between two slots, so that a fast warp's next write cannot overtake a slow warp's read.
      const int par = it & 1;
      ++it;
      const long long first_item = (long long)tile * p.KS;
      int b_first = 0, b_last = 0;
      if (!full_tile) {
        b_first = w4_owner(T, Gs, first_item);
        b_last = w4_owner(T, Gs, first_item + p.KS - 1);
        __threadfence();
      }
      w4g_epi_bar();
      if (warp == W4W_FIRST_EPI_WARP && lane == 0) {
        uint32_t ctrl = *abort_flag ? 1u : 0u;
        // split tile: count arrivals; the last contributor (found without waiting) adds the partial sums
        if (!ctrl && !full_tile && atomicAdd(counter(b_first), 1u) == (uint32_t)(b_last - b_first)) ctrl |= 2u;
        epi_flag[par] = ctrl;
      }
      w4g_epi_bar();
      const uint32_t ctrl = epi_flag[par];
      if (ctrl & 1u) break;
      if (ctrl & 2u) {
        __threadfence();
        const int rows = min(mt, p.M - m0);
#pragma unroll 1
        for (int c = 16 * e; c < rows; c += 32) {
          float sum[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) sum[u] = 0.0f;
#pragma unroll 1
          for (int o = b_first; o <= b_last; ++o) {  // fixed order: results do not depend on arrival order
            const int slot = partial_slot(o, w4_range_begin(T, Gs, o + 1) >= first_item + p.KS ? 0 : 1);
            const float* src = p.ws_partials + (size_t)slot * ((size_t)mt * W4_BN) + (size_t)c * W4_BN + nl;
            float v[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) v[u] = __ldcg(src + u * W4_BN);
#pragma unroll
            for (int u = 0; u < 16; ++u) sum[u] += v[u];
          }
#pragma unroll
          for (int u = 0; u < 16; u += 4)
            w4w_store_tokens4(p, Cout, m0 + c + u, n, lane, pack_out2<OUT_BF16>(sum[u], sum[u + 1]),
                              pack_out2<OUT_BF16>(sum[u + 2], sum[u + 3]));
        }
      }
    }
  } else if (warp >= W4W_FIRST_DQ_WARP) {
    // ------------------------------------------------------------------ dequant
    const int wd = warp - W4W_FIRST_DQ_WARP;
    const int q = warp & 3;       // TMEM lanes 32 q .. 32 q + 31, the quadrant this warp may touch
    const int j = wd >> 2;        // k 64 j .. 64 j + 63 of the slab: packed 16-byte chunks 2 j and 2 j + 1 of the row
    const int half = j >> 1;
    const int row = q * 32 + lane;
    const int sw = row & 7;
    const uint32_t off0 = row * 128 + (((2 * j) ^ sw) << 4);      // quarter-warps read 8 rows x 8 distinct chunks
    const uint32_t off1 = row * 128 + (((2 * j + 1) ^ sw) << 4);
    const uint32_t zero = ZT ? 0u : (uint32_t)p.zero;
    const uint32_t sub_lo = (0x6400u + zero) * 0x00010001u;                      // (1024 + zero) x2
    const uint32_t sub_hi = ((0x5400u + (zero << 4)) | 0x8000u) * 0x00010001u;   // -(64 + zero) x2
    const bool scaled = p.has_scales != 0;
    const int srow0 = (p.group <= W4_SLAB_K) ? (64 * j) / p.group : 0;
    const int srow1 = (p.group <= W4_SLAB_K) ? (64 * j + 32) / p.group : 0;
    const uint32_t st_addr = tmem_w + ((uint32_t)(q * 32) << 16) + (j & 1) * 32;
    int rs = 0, ws = half;        // a slab's halves go to stages 0, 1 and 2, 3 in turn
    uint32_t rphase = 0, wphase = 0;
    bool ok = true;
    while (ok && seg.next(tile, ks0, ks1)) {
#pragma unroll 1
      for (int ks = ks0; ks < ks1; ++ks) {
        if (!mbar_wait_warp(&raw_full[rs], rphase, ctl, ST_TIMEOUT_DEQUANT)) { ok = false; break; }
        const uint8_t* rawp = raw_base + rs * Cfg::RAW_BYTES;
        const uint4 v0 = *reinterpret_cast<const uint4*>(rawp + off0);
        const uint4 v1 = *reinterpret_cast<const uint4*>(rawp + off1);
        uint32_t s20 = 0x3C003C00u, s21 = 0x3C003C00u, z20 = 0u, z21 = 0u;
        if (scaled) {
          const __half* sS = reinterpret_cast<const __half*>(rawp + W4_RAW_PACKED);
          s20 = (uint32_t)__half_as_ushort(sS[srow0 * W4_BN + row]) * 0x00010001u;
          s21 = (uint32_t)__half_as_ushort(sS[srow1 * W4_BN + row]) * 0x00010001u;
        }
        if constexpr (ZT) {
          const __half* sZ = reinterpret_cast<const __half*>(rawp + W4_RAW_BYTES);
          z20 = (uint32_t)__half_as_ushort(sZ[srow0 * W4_BN + row]) * 0x00010001u;
          z21 = (uint32_t)__half_as_ushort(sZ[srow1 * W4_BN + row]) * 0x00010001u;
        }
        uint32_t o[32];
        w4_dequant8(v0.x, sub_lo, sub_hi, s20, !ZT && scaled, o + 0);
        w4_dequant8(v0.y, sub_lo, sub_hi, s20, !ZT && scaled, o + 4);
        w4_dequant8(v0.z, sub_lo, sub_hi, s20, !ZT && scaled, o + 8);
        w4_dequant8(v0.w, sub_lo, sub_hi, s20, !ZT && scaled, o + 12);
        w4_dequant8(v1.x, sub_lo, sub_hi, s21, !ZT && scaled, o + 16);
        w4_dequant8(v1.y, sub_lo, sub_hi, s21, !ZT && scaled, o + 20);
        w4_dequant8(v1.z, sub_lo, sub_hi, s21, !ZT && scaled, o + 24);
        w4_dequant8(v1.w, sub_lo, sub_hi, s21, !ZT && scaled, o + 28);
        if constexpr (ZT) {
#pragma unroll
          for (int i = 0; i < 32; ++i) w4_apply_zero(o[i], i < 16 ? s20 : s21, i < 16 ? z20 : z21, zero_mode);
        }
        // the packed bytes are in registers: hand the raw stage back to the producer
        __syncwarp();
        if (lane == 0) mbar_arrive(&raw_empty[rs]);
        if (++rs == RS) { rs = 0; rphase ^= 1u; }

        if (!mbar_wait_warp(&w_empty[ws], wphase ^ 1u, ctl, ST_TIMEOUT_DEQUANT)) { ok = false; break; }
        tc_fence_after_sync();
        tmem_st_32x32b_x32(st_addr + ws * W4W_W_COLS, o);
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) arrive_leader(&w_full[ws]);
        ws ^= 2;
        if (ws < 2) wphase ^= 1u;
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // neither CTA leaves while the other may still reach into it
  if (warp == 3) {
    tc_fence_after_sync();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace qg
