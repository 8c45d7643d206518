// W8A8 quantized (batched) matmul for sm_100a:
//   C[b, m, n] = cast( float(sum_k int32(A[b,m,k]) * int32(B[b,k,n])) [* scale_a[m]] * scale_b[n] )
//
// Persistent, warp-specialised kernel. One CTA per SM walks a list of 128 x BN output tiles:
//   warp 0      TMA producer: A tile [128 x 128 B] and B tile into a multistage shared-memory ring
//   warp 1      tcgen05.mma kind::i8 issuer; int32 accumulators live in tensor memory, double buffered
//   warps 2..9  epilogue: tcgen05.ld -> cvt.rn.f32.s32 -> fp32 scale(s) -> cvt.rn f16/bf16 -> staging tile -> bulk store; two
//               warps per 32 rows, each with half of the columns
// B is consumed in the operator's own [K, N] row-major layout as an MN-major operand (no transpose
// pass), or in [N, K] layout as a K-major operand.
#pragma once

#include "common.cuh"

namespace qg {

struct W8A8Params {
  const float* scale_b;
  const float* scale_a;  // nullable
  void* C;               // [batch, M, N] f16 / bf16
  int32_t* acc_out;      // nullable: raw int32 accumulators [batch, M, N]
  int batch, M, N, K;
  int sb_mode;  // 0: one value for all; 1: [N]; 2: [batch, N]
  int sa_mode;  // 0: none; 1: [M]; 2: [batch, M]
  int m_tiles, n_tiles, num_tiles, k_blocks;
  int group_m;  // tile rasterisation: the tiles of `group_m` row blocks are walked column block by column block

  int bn;            // columns per tile: the kernel's BN
  uint32_t* status;  // nullable device word
  unsigned long long wait_limit_ns;
  // Grouped (ragged) form: A and C are [M, K] / [M, N] stacks of row groups, B is [groups, ...]; row block i
  // of the table is (group, first row, valid rows <= 128).  Null for the plain and batched forms.
  const int* meta;
  int groups;
  int num_blocks;       // rows of the table
  int zero_uncovered;   // rows of C (16-bit outputs) that no block covers are set to zero
  // Tail split: work items from `split_from` on are half-width tiles (item split_from + 2i + h is the left or
  // right half of tile split_from + i), so that the last, partly filled round of the persistent grid keeps
  // twice as many SMs busy for about half as long.  num_items = num_tiles when nothing is split.
  int split_from, num_items;
  int early;      // let the next kernel on the stream set up beside this one (w8a8_impl says when)
  int withhold;   // test hook of the two-CTA form (qgemm_debug_withhold_commit)
  int tma_store;  // C is written with tiled bulk stores from a shared-memory staging tile
};

// One output tile's coordinates: batch index of B / scale_b, batch index of A / C / scale_a, first row, valid rows.
struct W8Tile {
  int bB, bA, m0, rows, n0, bn;  // n0: first column, bn: columns of this item
};

constexpr int W8_BM = 128;      // tile rows (= MMA M, one TMEM lane per row)
constexpr int W8_BK = 128;      // K bytes per pipeline stage (one 128-byte swizzle atom)
constexpr int W8_UMMA_K = 32;   // K per tcgen05.mma for 8-bit operands
constexpr int W8_EPI_WARPS = 8;
constexpr int W8_THREADS = (2 + W8_EPI_WARPS) * 32;

// How the CTAs of a launch share the work: each by itself; two cut a tile's K (see SPLITK below); or two make one tile of 256 x
// 256 with MMAs over both (see PAIR below).
enum W8Form { W8_ALONE, W8_SPLITK, W8_PAIR };

template <int BN, W8Form FORM = W8_ALONE>
struct W8Cfg {
  static constexpr int STAGES = (FORM == W8_PAIR || BN == 128) ? 6 : 4;
  static constexpr int A_BYTES = W8_BM * W8_BK;
  static constexpr int B_BYTES = (FORM == W8_PAIR ? BN / 2 : BN) * W8_BK;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TMEM_COLS = 2 * BN;
  static constexpr int BAR_BYTES = 256;
  static constexpr int SCALE_BYTES = W8_EPI_WARPS * 32 * 4;  // each epilogue warp's scales of 32 columns
  static constexpr int OUT_BYTES = W8_EPI_WARPS * 4096;      // each epilogue warp's staging tile: 32 rows x 64 outputs
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + OUT_BYTES + BAR_BYTES + SCALE_BYTES + 1024;  // + alignment slack
  static_assert(SMEM_BYTES <= 232448, "shared memory of a CTA");
};

__device__ __forceinline__ void w8_decode_tile(const W8A8Params& p, int tile, int& b, int& m_blk, int& n_blk) {
  const int per_batch = p.m_tiles * p.n_tiles;
  b = tile / per_batch;
  const int r = tile - b * per_batch;
  const int band = p.group_m * p.n_tiles;
  const int g = r / band;
  const int first_m = g * p.group_m;
  const int gsz = min(p.m_tiles - first_m, p.group_m);
  const int in_band = r - g * band;
  m_blk = first_m + in_band % gsz;
  n_blk = in_band / gsz;
}

template <bool PAIR>
__device__ __forceinline__ W8Tile w8_tile(const W8A8Params& p, int item, int crank) {
  int b, m_blk, n_blk;
  W8Tile t;
  if (item < p.split_from) {
    w8_decode_tile(p, item, b, m_blk, n_blk);
    t.n0 = n_blk * p.bn;
    t.bn = p.bn;
  } else {
    const int h = item - p.split_from;
    w8_decode_tile(p, p.split_from + (h >> 1), b, m_blk, n_blk);
    t.bn = p.bn >> 1;
    t.n0 = n_blk * p.bn + (h & 1) * t.bn;
  }
  if (p.meta == nullptr) {
    t.bB = t.bA = b;
    t.m0 = PAIR ? (2 * m_blk + crank) * W8_BM : m_blk * W8_BM;  // PAIR: a row block is 256 rows, 128 for each CTA
    t.rows = min(W8_BM, p.M - t.m0);
  } else {
    t.bB = ld_written(p.meta + 3 * m_blk);
    t.bA = 0;
    t.m0 = ld_written(p.meta + 3 * m_blk + 1);
    t.rows = min(ld_written(p.meta + 3 * m_blk + 2), W8_BM);
    // a table entry that points outside the tensors computes nothing (loads are bounds-checked by TMA)
    if (t.bB < 0 || t.bB >= p.groups || t.m0 < 0 || t.m0 >= p.M) { t.bB = 0; t.m0 = 0; t.rows = 0; }
    t.rows = min(t.rows, p.M - t.m0);
  }
  return t;
}

// Grouped form, rows of C that no table entry covers: set to zero by four of the epilogue warps before their first tile
// (they would otherwise wait for it), dealt to all CTAs; a launch that is sure to have such rows has a CTA on every SM,
// with or without a tile (w8a8_impl).  A clear of the whole output in front of the launch cost a pass over C (33 MB for
// 8192 x 2048: 8 us of 137) although normally every row is covered.  us, in the kernel / cleared in front: 4096 x 2048 with
// one open block of 32 19.0 / 24.2; 8192 x 1024, 16 blocks of 64 there could be 9.3 / 12.2; 65536 x 256 with one block of 100
// rows 12.2 / 15.5 (cleared by the two CTAs that have a tile: 935); 131072 x 1024 with 300 blocks of 20 rows 111 / 139.  (128 rows
// per CTA at a time, whatever M: 1055 x 2528 with three blocks 18.6 us instead of 9.8 cleared in front.)
__device__ __forceinline__ void w8_zero_uncovered(const W8A8Params& p, int warp4, int lane) {
  // A warp walks the table once per 32 rows, an entry per lane: which of the rows it covers.  Where there are not 128 rows
  // for every CTA the four warps take the same 32 rows, or 8, and share the columns.
  const bool own = p.M >= 128 * (long long)gridDim.x;
  const int chunk = own || p.M >= 32 * (long long)gridDim.x ? 32 : 8, step = own ? 4 * chunk : chunk;
  const int thread = own ? lane : warp4 * 32 + lane, threads = own ? 32 : 128;
  const int row_pieces = p.N / 8;  // N is a multiple of 16
  for (long long base = (long long)blockIdx.x * step + (own ? warp4 * 32 : 0); base < p.M; base += (long long)gridDim.x * step) {
    const int row0 = (int)base, n_here = min(chunk, p.M - row0);
    const uint32_t all_rows = n_here == 32 ? 0xffffffffu : (1u << n_here) - 1u;
    uint32_t open_rows = all_rows;
    for (int i = lane; open_rows != 0 && i - lane < p.num_blocks; i += 32) {
      uint32_t mine = 0;
      if (i < p.num_blocks) {
        const int g = ld_written(p.meta + 3 * i), first = ld_written(p.meta + 3 * i + 1);
        const int rows = min(ld_written(p.meta + 3 * i + 2), W8_BM);
        if (g >= 0 && g < p.groups && first >= 0 && first < p.M && rows > 0) {  // as in w8_tile
          const int lo = max(first - row0, 0), hi = min(first - row0 + rows, 32);
          if (lo < hi) mine = (hi - lo == 32 ? 0xffffffffu : (1u << (hi - lo)) - 1u) << lo;
        }
      }
      open_rows &= ~__reduce_or_sync(0xffffffffu, mine);
    }
    uint4* const dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.C) + (size_t)base * (size_t)p.N);
    if (open_rows == all_rows) {
      const long long pieces = (long long)n_here * row_pieces;
#pragma unroll 4
      for (long long c = thread; c < pieces; c += threads) dst[c] = make_uint4(0u, 0u, 0u, 0u);
      continue;
    }
    while (open_rows) {
      const int r = __ffs(open_rows) - 1;
      open_rows &= open_rows - 1;
      for (int c = thread; c < row_pieces; c += threads) dst[(size_t)r * row_pieces + c] = make_uint4(0u, 0u, 0u, 0u);
    }
  }
}

// SPLITK is the form for weights [K, N] and a very long K on grids that would leave half of the SMs idle (w8a8_impl): the kernel is
// launched in clusters of two CTAs, one tile per cluster; each CTA accumulates
// one half of the K range in its own tensor memory; then each CTA writes its int32 accumulators of the OTHER CTA's
// half of the columns into that CTA's shared memory (the pipeline stages, idle by then) through distributed shared
// memory, adds what it received to its own half and runs the epilogue for that half - an exact integer sum, so the
// result is bit-identical to the unsplit kernel's, the exchange runs in both directions at once and each CTA
// converts and stores half a tile.  The counterpart in the
// reference is the K split of examples/gemm_splitk/example_tilelang_gemm_splitk.py:15-48, whose partial tiles meet
// in global memory through atomic adds (src/tl_templates/ascend/common.h:249-259).
//
// PAIR: a cluster of two CTAs makes tiles of 256 x 256 with MMAs over both (tcgen05.mma.cta_group::2): CTA r holds rows 128 r ..
// of A and of the accumulator, and loads half of the columns of B, which the tensor cores of both read.  A k block costs each
// CTA 32 KB of loads instead of 48, so that six of them are in flight instead of four, and B crosses from L2 once for 256 rows.
// The leader (rank 0) issues; all bytes are counted on its barriers; its commits signal both CTAs, and the epilogue warps of both
// hand an accumulator back to it.  Traffic is what bounds these shapes, for what it costs in time and, at the power limit, in
// clock: 4096 x 4096 x 14336 166 -> 148 us (3.2 POPS, cuBLASLt's plain int8 GEMM 3.0; tensor pipe 92 % of active cycles instead of
// 79, 1.9 GB from L2 into the SMs instead of 2.8), 16 x 512 x 7168 x 2048 [N, K] 101 -> 89.  Which shapes take it: w8_pair_pays in qgemm_api.cu.
template <int BN, bool B_NK, bool OUT_BF16, W8Form FORM = W8_ALONE>
__global__ void __launch_bounds__(W8_THREADS, 1)
w8a8_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmC, const W8A8Params p) {
  using Cfg = W8Cfg<BN, FORM>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr bool SPLITK = FORM == W8_SPLITK, PAIR = FORM == W8_PAIR;
  static_assert(!(SPLITK && B_NK), "K is cut for weights [K, N] only");
  // Two warps share the columns of 32 rows and store them in pieces of 64: an item of 128 columns at least (a half-width one, or
  // a CTA's half of a tile whose K is cut, comes from 256).
  static_assert(BN == 128 || (BN == 256 && (BN / 2) % 128 == 0), "columns of a tile");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_stage = smem + STAGES * Cfg::STAGE_BYTES;  // 1024-byte aligned: 128-byte swizzled staging tiles
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_stage + Cfg::OUT_BYTES);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* drain = tempty + 2;
  uint64_t* stages_free = drain + 1;    // split form: the peer's MMAs have finished reading the peer's stages
  uint64_t* partial_full = drain + 2;   // split form: the peer's accumulators for this CTA's columns have arrived
  uint64_t* reported = drain + 3;       // two-CTA tiles: the second CTA's producer has ended (pair_wait_copies)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 4);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  uint32_t* peer_issued = tmem_slot + 2;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // split form: CTA `crank` of the pair takes the k blocks [kb_begin, kb_end) of tile (block index / 2)
  const int crank = FORM != W8_ALONE ? (int)cluster_ctarank() : 0;
  const int tile_first = FORM != W8_ALONE ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int tile_stride = FORM != W8_ALONE ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int kb_begin = SPLITK ? (crank ? p.k_blocks / 2 : 0) : 0;
  const int kb_end = SPLITK ? (crank ? p.k_blocks : p.k_blocks / 2) : p.k_blocks;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(stages_free, W8_EPI_WARPS);
    mbar_init(partial_full, W8_EPI_WARPS);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull[i], 1);
      mbar_init(&tempty[i], (PAIR ? 2 : 1) * W8_EPI_WARPS);  // PAIR: both CTAs', on the leader's barrier
    }
    if (p.tma_store) tma_prefetch_desc(&tmC);
    mbar_init(drain, 1);
    mbar_init(reported, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if constexpr (FORM != W8_ALONE) cluster_sync_all();  // both CTAs' barriers exist before either signals the other's
  else __syncthreads();
  // Launched as a programmatic dependent: set up beside the end of the kernel in front (the quantiser and the W8A8 kernels let
  // theirs start early), but nothing is read, written or taken from the SM's tensor memory before that kernel is done.  Then the
  // next kernel may set up beside this one.  The first loads do not wait for the tensor memory.
  pdl_wait();
  if (p.early) pdl_launch_dependents();
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
      tmem_relinquish();
    }
  }
  uint32_t tmem_base = 0;
  if (warp != 0) {
    tc_fence_before_sync();
    asm volatile("bar.sync 1, %0;" ::"n"(W8_THREADS - 32) : "memory");
    tc_fence_after_sync();
    tmem_base = *tmem_slot;
  }
  const WaitCtl ctl{abort_flag, p.status, p.wait_limit_ns};

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0, issued_mask = 0, parity_mask = 0, fills = 0;
      bool ok = true;
      const bool idle = PAIR && p.withhold == 3 + crank && tile_first == tile_stride - 1;  // test hook: this CTA copies nothing
      for (int tile = idle ? p.num_items : tile_first; ok && tile < p.num_items; tile += tile_stride) {
        const W8Tile t = w8_tile<PAIR>(p, tile, crank);
        const int m0 = t.m0, n0 = t.n0;
        const int b_boxes = B_NK ? 1 : (t.bn + 127) / 128;  // 128-column boxes of B actually needed
        const uint32_t tx = Cfg::A_BYTES + (B_NK ? (uint32_t)Cfg::B_BYTES : (uint32_t)(b_boxes * W8_BK * 128));
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1u, ctl, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
          uint8_t* sA = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* sB = sA + Cfg::A_BYTES;
          if constexpr (PAIR) {
            // both CTAs' bytes are counted on the leader's barrier; columns: this CTA's half of the item's
            const uint32_t bar = mapa_u32(smem_u32(&full[stage]), 0);
            const int nh = n0 + crank * (t.bn >> 1);
            if (crank == 0) mbar_arrive_expect_tx(&full[stage], 2 * Cfg::STAGE_BYTES);
            tma_load_3d_pair(sA, &tmA, bar, kb * W8_BK, m0, t.bA);
            if constexpr (B_NK) tma_load_3d_pair(sB, &tmB, bar, kb * W8_BK, nh, t.bB);
            else tma_load_3d_pair(sB, &tmB, bar, nh, kb * W8_BK, t.bB);
            ++fills;
            if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            continue;
          }
          mbar_arrive_expect_tx(&full[stage], tx);
          tma_load_3d(sA, &tmA, &full[stage], kb * W8_BK, m0, t.bA);
          if constexpr (B_NK) {
            tma_load_3d(sB, &tmB, &full[stage], kb * W8_BK, n0, t.bB);
          } else {
#pragma unroll
            for (int c = 0; c < BN / 128; ++c)
              if (c < b_boxes) tma_load_3d(sB + c * (W8_BK * 128), &tmB, &full[stage], n0 + c * 128, kb * W8_BK, t.bB);
          }
          issued_mask |= 1u << stage;
          parity_mask = (parity_mask & ~(1u << stage)) | (phase << stage);
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if constexpr (PAIR) {
        pair_wait_copies(full, STAGES, Cfg::STAGE_BYTES, fills, crank, reported, peer_issued, ctl);
      } else if (!ok) {
        // Gave up: wait (bounded) until every bulk copy already issued has landed before the CTA may exit.
        for (int s = 0; s < STAGES; ++s) {
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
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer (PAIR: the leader's, for both CTAs)
    // The warp runs converged and one hardware-elected lane issues, which lets the compiler keep the descriptors in uniform
    // registers.  The stage descriptors differ by their start address only.
    constexpr uint32_t K_STEP = (B_NK ? W8_UMMA_K : W8_UMMA_K * 128) >> 4;  // B's start address from one MMA to the next
    // K-major: 128 bytes of K per row.  [K rows][128 B of N]: 32 K rows per MMA = 4096 B; the next 128 columns are one
    // box (16 KB) further.
    const uint64_t b_desc = B_NK ? make_desc_kmajor(0) : make_desc_mnmajor(0, W8_BK * 128);
    const uint64_t a_desc = make_desc_kmajor(0);
    const uint32_t smem0 = smem_u32(smem);
    int stage = 0;
    uint32_t phase = 0;
    int it = 0;
    bool ok = true;
    for (int tile = PAIR && crank != 0 ? p.num_items : tile_first; ok && tile < p.num_items; tile += tile_stride, ++it) {
      const uint32_t bn = (uint32_t)((tile < p.split_from) ? p.bn : (p.bn >> 1));
      const uint32_t idesc = make_idesc(ACC_S32, FMT_S8, FMT_S8, 0, B_NK ? 0 : 1, PAIR ? 2 * W8_BM : W8_BM, bn);
      const int buf = it & 1;
      const uint32_t tphase = (it >> 1) & 1;
      if (!mbar_wait_warp(&tempty[buf], tphase ^ 1u, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
      tc_fence_after_sync();
      const uint32_t d = tmem_base + buf * BN;
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!mbar_wait_warp(&full[stage], phase, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
        tc_fence_after_sync();
        if (elect_one_sync()) {
          const uint32_t sA = smem0 + stage * Cfg::STAGE_BYTES;
          const uint64_t adesc = a_desc | (uint64_t)((sA & 0x3FFFFu) >> 4);
          const uint64_t bdesc = b_desc | (uint64_t)(((sA + Cfg::A_BYTES) & 0x3FFFFu) >> 4);
#pragma unroll
          for (int k = 0; k < W8_BK / W8_UMMA_K; ++k) {
            const uint64_t ad = adesc + (uint64_t)(k * (W8_UMMA_K >> 4)), bd = bdesc + (uint64_t)(k * K_STEP);
            if constexpr (PAIR) umma_i8_ss_pair(d, ad, bd, idesc, (kb | k) != 0 ? 1u : 0u);
            else umma_i8_ss(d, ad, bd, idesc, ((kb - kb_begin) | k) != 0 ? 1u : 0u);
          }
          if constexpr (PAIR) umma_commit_pair(&empty[stage]);
          else umma_commit(&empty[stage]);
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
      if (ok && elect_one_sync()) {  // the elected lane is the same one every time
        if constexpr (PAIR) {
          const bool withheld = p.withhold == 1 && tile_first == tile_stride - 1 && tile + tile_stride >= p.num_items;
          if (!withheld) umma_commit_pair(&tfull[buf]);
        } else {
          umma_commit(&tfull[buf]);
        }
      }
    }
    if (!ok) {
      if (elect_one_sync()) {
        if constexpr (PAIR) umma_commit_pair(drain);
        else umma_commit(drain);
      }
      if (lane == 0) {
        const uint64_t t0 = global_timer_ns();
        while (!mbar_try_wait(drain, 0)) {
          if (global_timer_ns() - t0 > p.wait_limit_ns) break;
        }
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    // A warp keeps the next 32-column chunk's tcgen05.ld and column scales (a scale per lane, handed round through 128 bytes of
    // shared memory) in flight while it converts and stores the current one.  With four warps a tile of 128 x 256 took 6 us
    // from the end of its MMAs, more than its MMAs below K = 2048, and as much again at the end of every launch:
    // 4096 x 1024 x 4096 29.0 -> 20.9 us, 3000 x 1024 x 1024 12.3 -> 10.3, 512 x 512 x 4096 8.2 -> 7.2, 4000 rows in 32 groups,
    // K = 1024, N = 4096 52.7 -> 43.1; K = 4096 and more as before (the power limit).
    const int q = warp & 3;         // TMEM lane quadrant this warp may read
    const int e = (warp - 2) >> 2;  // which half of the columns
    const uint64_t pol_out = l2_policy_evict_first();  // the output is written once and not read here
    float* sb_s = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + Cfg::BAR_BYTES) + (warp - 2) * 32;
    uint8_t* my_stage = out_stage + (warp - 2) * 4096;  // [32 rows][128 B], 16-byte piece j of row r at (j ^ (r & 7))
    int it = 0;
    if (p.zero_uncovered && e == 0) w8_zero_uncovered(p, q, lane);
    // split form: the other CTA's accumulators travel through CTA 0's pipeline stages, one 16-byte piece per
    // (row, four columns): piece (col / 4, row) at ((col / 4) * 128 + row) * 16, so that a warp's 32 rows are
    // 512 contiguous bytes for the sender's stores and the receiver's loads alike
    const uint32_t part_row = smem_u32(smem) + (uint32_t)(q * 32 + lane) * 16u;
    for (int tile = tile_first; tile < p.num_items; tile += tile_stride, ++it) {
      const W8Tile t = w8_tile<PAIR>(p, tile, crank);
      const int buf = it & 1;
      const uint32_t tphase = (it >> 1) & 1;
      const int m = t.m0 + q * 32 + lane;
      const bool row_ok = q * 32 + lane < t.rows;
      float sa = 1.0f;
      if (p.sa_mode != 0 && row_ok) sa = ld_written(p.scale_a + (p.sa_mode == 2 ? (size_t)t.bA * p.M : 0) + m);
      const float* sbp = p.scale_b + (p.sb_mode == 2 ? (size_t)t.bB * p.N : 0);
      auto column_scale = [&](int c) {  // of this lane's column of chunk c
        const int n = t.n0 + c * 32 + lane;
        return p.C == nullptr ? 0.f : (p.sb_mode == 0 ? ld_written(sbp) : (n < p.N ? ld_written(sbp + n) : 0.f));
      };
      // This warp's chunks of 32 columns.  Split form: of the half of the tile that this CTA finishes.
      const int own_chunks = (SPLITK ? t.bn >> 6 : t.bn >> 5) >> 1;
      const int c_begin = (SPLITK ? crank * (t.bn >> 6) : 0) + e * own_chunks, chunks = c_begin + own_chunks;
      float sb_next = column_scale(c_begin);
      if (!mbar_wait_warp(&tfull[buf], tphase, ctl, ST_TIMEOUT_EPILOGUE)) break;
      tc_fence_after_sync();
      // Split form: each CTA of the pair finishes ONE half of the tile's columns (CTA r: columns r * bn/2 ...): it sends
      // its accumulators of the other half into the peer's pipeline stages and receives the peer's for its own, so
      // that the exchange runs in both directions at once and each CTA converts and stores half a tile.
      if constexpr (SPLITK) {
        const uint32_t taddr_s = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN;
        const uint32_t peer = (uint32_t)(crank ^ 1);
        const int peer_begin = (int)peer * (t.bn >> 6) + e * own_chunks;  // the chunks that this warp sends
        // this CTA's MMAs are done (tfull): the peer may write into its stages
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(stages_free), peer));
        // ... and the peer's are done when its epilogue warps have said so here
        if (!mbar_wait_warp(stages_free, 0, ctl, ST_TIMEOUT_EPILOGUE)) break;
        const uint32_t dst_row = mapa_u32(part_row, peer);
#pragma unroll 1
        for (int c = 0; c < own_chunks; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr_s + (peer_begin + c) * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int jj = 0; jj < 8; ++jj)
            st_cluster_v4(dst_row + (uint32_t)(((e * own_chunks + c) * 8 + jj) * 128 * 16), r[4 * jj], r[4 * jj + 1], r[4 * jj + 2], r[4 * jj + 3]);
        }
        fence_acq_rel_cluster();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(partial_full), peer));
        // the peer's sums for this CTA's half
        bool got = true;
        if (lane == 0) {
          const uint64_t t0 = global_timer_ns();
          while (!mbar_try_wait_cluster(partial_full, 0)) {
            if (*abort_flag || global_timer_ns() - t0 > p.wait_limit_ns) {
              *abort_flag = 1u;
              if (p.status) atomicMax(p.status, (uint32_t)ST_TIMEOUT_EPILOGUE);
              got = false;
              break;
            }
          }
        }
        got = __shfl_sync(0xffffffffu, got ? 1 : 0, 0) != 0;
        if (!got) break;
        fence_acq_rel_cluster();
      }
      const size_t row_off = ((size_t)t.bA * p.M + (row_ok ? m : 0)) * (size_t)p.N;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * BN;
      // Whole row blocks go out as tiled bulk stores (coalesced, clipped at the tensor's edge); a partial
      // block of the grouped form must not touch the rows after it and uses per-row stores.
      const bool tma_out = p.tma_store != 0 && (p.meta == nullptr || t.rows == W8_BM);
      uint32_t r[2][32];
      tmem_ld_32x32b_x32(taddr + c_begin * 32, r[0]);
#pragma unroll 1
      for (int c2 = c_begin; c2 < chunks; c2 += 2) {
        if (tma_out) {  // the previous bulk store has read the staging tile
          if (lane == 0) bulk_wait_group_read0();
          __syncwarp();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = c2 + h;
          if (c >= chunks) break;
          __syncwarp();  // the previous chunk's reads of sb_s are done
          sb_s[lane] = sb_next;
          __syncwarp();
          if (c + 1 < chunks) sb_next = column_scale(c + 1);
          tmem_ld_wait();                                                     // chunk c is in r[h]
          if (c + 1 < chunks) tmem_ld_32x32b_x32(taddr + (c + 1) * 32, r[h ^ 1]);  // chunk c + 1 in flight
          if constexpr (SPLITK) {  // add the other CTA's half of the K range (exact: int32)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint4 pv;
              asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                           : "=r"(pv.x), "=r"(pv.y), "=r"(pv.z), "=r"(pv.w)
                           : "r"(part_row + (uint32_t)(((c - crank * (t.bn >> 6)) * 8 + j) * 128 * 16)));
              r[h][4 * j] += pv.x;
              r[h][4 * j + 1] += pv.y;
              r[h][4 * j + 2] += pv.z;
              r[h][4 * j + 3] += pv.w;
            }
          }
          const int n = t.n0 + c * 32;
          if (row_ok && n < p.N && p.acc_out != nullptr) {
            int4* dst = reinterpret_cast<int4*>(p.acc_out + row_off + n);
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (n + 4 * j < p.N)
                dst[j] = make_int4((int)r[h][4 * j], (int)r[h][4 * j + 1], (int)r[h][4 * j + 2], (int)r[h][4 * j + 3]);
          }
          if (tma_out) {
            if (n < p.N) {
              const float4* sv = reinterpret_cast<const float4*>(sb_s);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float4 s_lo = sv[2 * j], s_hi = sv[2 * j + 1];
                const float sc[8] = {s_lo.x, s_lo.y, s_lo.z, s_lo.w, s_hi.x, s_hi.y, s_hi.z, s_hi.w};
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const int col = 8 * j + 2 * e;
                  float f0 = __int2float_rn((int)r[h][col]), f1 = __int2float_rn((int)r[h][col + 1]);
                  if (p.sa_mode != 0) { f0 = __fmul_rn(f0, sa); f1 = __fmul_rn(f1, sa); }
                  f0 = __fmul_rn(f0, sc[2 * e]);
                  f1 = __fmul_rn(f1, sc[2 * e + 1]);
                  o[e] = pack_out2<OUT_BF16>(f0, f1);
                }
                *reinterpret_cast<uint4*>(my_stage + lane * 128 + (((h * 4 + j) ^ (lane & 7)) << 4)) =
                    make_uint4(o[0], o[1], o[2], o[3]);
              }
            }
          } else if (row_ok && n < p.N) {
            if (p.C != nullptr) {
              uint16_t* cbase = reinterpret_cast<uint16_t*>(p.C) + row_off + n;
              const float4* sv = reinterpret_cast<const float4*>(sb_s);
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (n + 8 * j < p.N) {
                  const float4 s_lo = sv[2 * j], s_hi = sv[2 * j + 1];
                  const float sc[8] = {s_lo.x, s_lo.y, s_lo.z, s_lo.w, s_hi.x, s_hi.y, s_hi.z, s_hi.w};
                  uint32_t o[4];
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const int col = 8 * j + 2 * e;
                    float f0 = __int2float_rn((int)r[h][col]), f1 = __int2float_rn((int)r[h][col + 1]);
                    if (p.sa_mode != 0) { f0 = __fmul_rn(f0, sa); f1 = __fmul_rn(f1, sa); }
                    f0 = __fmul_rn(f0, sc[2 * e]);
                    f1 = __fmul_rn(f1, sc[2 * e + 1]);
                    o[e] = pack_out2<OUT_BF16>(f0, f1);
                  }
                  *reinterpret_cast<uint4*>(cbase + 8 * j) = make_uint4(o[0], o[1], o[2], o[3]);
                }
              }
            }
          }
        }
        if (tma_out && t.n0 + c2 * 32 < p.N && t.m0 + q * 32 < p.M) {  // a box wholly outside is not issued
          fence_proxy_async_smem();  // this thread's staging writes are visible to the bulk-copy engine
          __syncwarp();
          if (lane == 0) {
            tma_store_3d_hint(&tmC, my_stage, t.n0 + c2 * 32, t.m0 + q * 32, t.bA, pol_out);
            bulk_commit_group();
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_leader(&tempty[buf]);
        else mbar_arrive(&tempty[buf]);
      }
    }
    if (lane == 0) bulk_wait_group_read0();  // the staging tile must outlive the last bulk store's read
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if constexpr (FORM != W8_ALONE) cluster_sync_all();  // neither CTA of the pair leaves while the other may still reach into it
  if (warp == 1) {
    tc_fence_after_sync();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
    else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

}  // namespace qg
