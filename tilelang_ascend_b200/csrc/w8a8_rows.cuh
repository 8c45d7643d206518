// W8A8 quantized (batched) matmul for few tokens, sm_100a: the weights are the MMA's M operand.
//   C[b, m, n] = cast( float(sum_k int32(A[b,m,k]) * int32(B[b,k,n])) [* scale_a[m]] * scale_b[n] ), as in w8a8.cuh
//
// Few tokens make the product a stream of the weights, so what counts is how many SMs load and how much each has in
// flight.  w8a8.cuh gives a 128-token row block to one CTA per 128 or 256 columns: 112 CTAs (14336 columns), 64 (8192) or 32
// (4096) of one tile each, whose pipeline fill, int32 exchange and store follow one another.  Here a tile is 128 weight
// columns x up to 128 tokens and K is cut over a cluster of S = 1, 2, 4 or 8 CTAs, one CTA per SM where that is enough, with most of
// the SM's shared memory as its pipeline (w8_rows_plan).  24 tokens, K = 4096, N = 14336: 22.6 us by w8a8.cuh, 14.7 with two CTAs
// per SM and a pipeline of 96 KB each, now 13.6 (58.7 MB at 6.5 TB/s: 9), each as one graph; with the quantiser in front, calls one
// after another, 28.7, 19.1, now 15.9; 8192 x 8192, 128 tokens 20.7 -> 18.5.  What is left is the start of the launch, the pipeline's
// first loads and the two cluster barriers.
//   warp 0      TMA: [128 columns x 128 k] of weights ([N, K]: K-major rows; [K, N]: MN-major) and [tokens x 128 k] of A
//   warp 1      tcgen05.mma kind::i8 (M = 128 weight columns, N = tokens rounded up to 16), allocates tensor memory
//   warps 2..5  epilogue
// The CTAs of a cluster then share the tokens: each writes its int32 sums of the others' tokens into their (idle) pipeline
// stages through distributed shared memory, adds what it received for its own (exact) and converts and stores those.
// All threads of a cluster meet at the two cluster barriers whatever happened before: a wait that gave up only sets the
// CTA's abort flag, so no barrier is ever left open.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "w8a8.cuh"

namespace qg {

constexpr int W8R_THREADS = 192;
constexpr int W8R_MAX_MT = 128;
constexpr int W8R_MAX_SPLIT = 8;
constexpr int W8R_RING_BYTES = 96 * 1024;       // two CTAs per SM
constexpr int W8R_RING_BYTES_ONE = 208 * 1024;  // one
constexpr int W8R_MAX_STAGES = 12;
constexpr int W8R_W_BYTES = 128 * 128;
constexpr int W8R_EXTRA_BYTES = 256 + 1024;  // barriers, alignment slack
static_assert(W8R_RING_BYTES_ONE + W8R_EXTRA_BYTES <= 232448 && 8 * (2 * W8R_MAX_STAGES + 2) + 8 <= 256, "shared memory of a CTA");

struct W8RowsParams {
  const float* scale_b;
  const float* scale_a;  // nullable
  void* C;               // [batch, M, N] f16 / bf16
  int M, N;
  int sb_mode, sa_mode;  // as in W8A8Params
  int n_tiles, m_tiles, k_blocks;
  int mt;                // tokens per tile: M rounded up to 16, at least 4 per CTA of the cluster
  int tmem_cols;         // power of two >= max(mt, 32)
  int ring;              // bytes of the pipeline's stages
  uint32_t* status;
  unsigned long long wait_limit_ns;
};

template <bool B_NK, bool OUT_BF16>
__global__ void __launch_bounds__(W8R_THREADS, 2)
w8a8_rows_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const W8RowsParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + p.ring);
  uint64_t* empty = full + W8R_MAX_STAGES;
  uint64_t* tfull = empty + W8R_MAX_STAGES;
  uint64_t* drain = tfull + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int S = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
  const int mt = p.mt;
  const int stage_bytes = W8R_W_BYTES + mt * 128;
  const int stages = min(W8R_MAX_STAGES, p.ring / stage_bytes);
  const int tile = (int)blockIdx.x / S;
  const int b = tile / (p.n_tiles * p.m_tiles);
  const int in_b = tile - b * (p.n_tiles * p.m_tiles);
  const int n0 = in_b / p.m_tiles * 128, m0 = in_b % p.m_tiles * mt;  // neighbouring tiles share the weights
  const int kb0 = (int)((long long)p.k_blocks * rank / S), kb1 = (int)((long long)p.k_blocks * (rank + 1) / S);

  if (threadIdx.x == 0) {
    for (int s = 0; s < W8R_MAX_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  // Launched as a programmatic dependent: resident beside the end of the kernel in front (the activation quantiser lets its
  // dependents start early), but nothing is read, written or taken from the SM's tensor memory before that kernel is done.
  // Then the next kernel may set up beside this one (the quantiser and this kernel wait for this whole grid before they touch
  // anything): 1 x 2048 x 2048 4.9 -> 4.2 us a call, 64 x 1024 x 1024 5.2 -> 4.6, 256 x 1024 x 1024 6.5 -> 6.2, each as one graph.
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();
  if (warp == 1) {
    tmem_alloc(tmem_slot, (uint32_t)p.tmem_cols);
    tmem_relinquish();
  }
  uint32_t tmem_base = 0;
  if (warp != 0) {  // the first loads do not wait for the tensor memory (256 x 1024 x 1024 by this form 6.15 -> 5.81 us)
    tc_fence_before_sync();
    asm volatile("bar.sync 1, %0;" ::"n"(W8R_THREADS - 32) : "memory");
    tc_fence_after_sync();
    tmem_base = *tmem_slot;
  }
  const WaitCtl ctl{abort_flag, p.status, p.wait_limit_ns};
  const int q = warp & 3;
  const int nl = q * 32 + lane;  // weight column inside the tile == TMEM lane
  bool ok = true;
  if (warp == 0) {
    // ------------------------------------------------------------------ producer
    if (lane == 0) {
      int st = 0;
      uint32_t phase = 0, issued_mask = 0, parity_mask = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty[st], phase ^ 1u, ctl, ST_TIMEOUT_PRODUCER)) { ok = false; break; }
        uint8_t* dst = smem + st * stage_bytes;
        mbar_arrive_expect_tx(&full[st], (uint32_t)stage_bytes);
        if constexpr (B_NK) tma_load_3d(dst, &tmB, &full[st], kb * 128, n0, b);
        else tma_load_3d(dst, &tmB, &full[st], n0, kb * 128, b);
        tma_load_3d(dst + W8R_W_BYTES, &tmA, &full[st], kb * 128, m0, b);
        issued_mask |= 1u << st;
        parity_mask = (parity_mask & ~(1u << st)) | (phase << st);
        if (++st == stages) { st = 0; phase ^= 1u; }
      }
      if (!ok) {  // wait (bounded) for the copies still in flight
        for (int s = 0; s < stages; ++s) {
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
    // ------------------------------------------------------------------ MMA issuer (converged warp, one elected lane)
    const uint32_t idesc = make_idesc(ACC_S32, FMT_S8, FMT_S8, B_NK ? 0 : 1, 0, 128, mt);
    constexpr uint32_t W_STEP = (B_NK ? W8_UMMA_K : W8_UMMA_K * 128) >> 4;
    const uint64_t wdesc0 = B_NK ? make_desc_kmajor(0) : make_desc_mnmajor(0, W8R_W_BYTES);
    const uint64_t adesc0 = make_desc_kmajor(0);
    const uint32_t smem0 = smem_u32(smem);
    int st = 0;
    uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full[st], phase, ctl, ST_TIMEOUT_MMA)) { ok = false; break; }
      tc_fence_after_sync();
      if (elect_one_sync()) {
        const uint32_t sW = smem0 + st * stage_bytes;
        const uint64_t wdesc = wdesc0 | (uint64_t)((sW & 0x3FFFFu) >> 4);
        const uint64_t adesc = adesc0 | (uint64_t)(((sW + W8R_W_BYTES) & 0x3FFFFu) >> 4);
#pragma unroll
        for (int k = 0; k < W8_BK / W8_UMMA_K; ++k)
          umma_i8_ss(tmem_base, wdesc + (uint64_t)(k * W_STEP), adesc + (uint64_t)(k * (W8_UMMA_K >> 4)), idesc,
                     ((kb - kb0) | k) != 0 ? 1u : 0u);
        umma_commit(&empty[st]);
      }
      if (++st == stages) { st = 0; phase ^= 1u; }
    }
    if (elect_one_sync()) umma_commit(ok ? tfull : drain);
    if (!ok && lane == 0) {
      const uint64_t t0 = global_timer_ns();
      while (!mbar_try_wait(drain, 0)) {
        if (global_timer_ns() - t0 > p.wait_limit_ns) break;
      }
    }
  } else {
    ok = mbar_wait_warp(tfull, 0, ctl, ST_TIMEOUT_EPILOGUE);  // all of this CTA's MMAs
    tc_fence_after_sync();
  }
  __syncwarp();

  // ------------------------------------------------------------------ exchange and epilogue
  const int mine = mt / S;  // tokens this CTA finishes: [rank * mine, (rank + 1) * mine), a multiple of 4
  const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16);
  // a peer's sums: [sender (rank without the receiver)][token][128 columns] int32, in the receiver's pipeline stages
  // in pieces of 16 tokens where the share allows it (their loads overlap; a serial chain of pieces of 4 cost 100 tokens in one
  // CTA 4 us), else of 4
  auto send = [&](auto piece) {
    constexpr int CH = decltype(piece)::value;
    for (int d = 1; d < S; ++d) {
      const int to = (rank + d) % S;
      const int slot = rank < to ? rank : rank - 1;
      const uint32_t dst = mapa_u32(smem_u32(smem) + (uint32_t)((slot * mine * 128 + nl) * 4), (uint32_t)to);
#pragma unroll 1
      for (int c = 0; c < mine; c += CH) {
        uint32_t r[CH];
        if constexpr (CH == 16) tmem_ld_32x32b_x16(taddr + to * mine + c, r);
        else tmem_ld_32x32b_x4(taddr + to * mine + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < CH; ++j)
          asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst + (uint32_t)((c + j) * 512)), "r"(r[j]) : "memory");
      }
    }
  };
  const int n = n0 + nl;
  float sb = 0.f;
  if (warp >= 2 && n < p.N) sb = ld_written(p.scale_b + (p.sb_mode == 0 ? 0 : (p.sb_mode == 2 ? (size_t)b * p.N : 0) + n));
  const float* sap = p.scale_a + (p.sa_mode == 2 ? (size_t)b * p.M : 0);
  auto finish = [&](auto piece) {
    constexpr int CH = decltype(piece)::value;
    uint16_t* Cout = reinterpret_cast<uint16_t*>(p.C) + (size_t)b * p.M * p.N;
    const int* got = reinterpret_cast<const int*>(smem) + nl;
#pragma unroll 1
    for (int c = 0; c < mine; c += CH) {
      const int col0 = rank * mine + c, m = m0 + col0;
      if (m >= p.M) break;
      uint32_t r[CH];
      if constexpr (CH == 16) tmem_ld_32x32b_x16(taddr + col0, r);
      else tmem_ld_32x32b_x4(taddr + col0, r);
      float sa[CH];
      if (p.sa_mode != 0) {
#pragma unroll
        for (int j = 0; j < CH; ++j) sa[j] = m + j < p.M ? ld_written(sap + m + j) : 0.f;
      }
      tmem_ld_wait();
#pragma unroll 1
      for (int s = 0; s < S - 1; ++s)
#pragma unroll
        for (int j = 0; j < CH; ++j) r[j] += (uint32_t)got[(s * mine + c + j) * 128];
#pragma unroll
      for (int j = 0; j < CH; j += 4) {
        float f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          f[i] = __int2float_rn((int)r[j + i]);
          if (p.sa_mode != 0) f[i] = __fmul_rn(f[i], sa[j + i]);
          f[i] = __fmul_rn(f[i], sb);
        }
        int row = m + j, col = n;
        const uint2 v = transpose_tokens4(lane, pack_out2<OUT_BF16>(f[0], f[1]), pack_out2<OUT_BF16>(f[2], f[3]), row, col);
        if (row < p.M && col < p.N) *reinterpret_cast<uint2*>(Cout + (size_t)row * p.N + col) = v;
      }
    }
  };
  constexpr std::integral_constant<int, 16> P16{};
  constexpr std::integral_constant<int, 4> P4{};
  if (S > 1) {
    cluster_sync_all();  // every CTA's MMAs have read their stages
    if (warp >= 2 && ok) {
      if (mine % 16 == 0) send(P16);
      else send(P4);
    }
    cluster_sync_all();  // release / acquire: what the peers sent is here, and nobody writes to a peer any more
  }
  if (warp >= 2 && ok) {
    if (mine % 16 == 0) finish(P16);
    else finish(P4);
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

}  // namespace qg
