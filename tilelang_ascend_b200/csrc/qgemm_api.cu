// Host side of libqgemm.so: argument validation, TMA tensor-map encoding, kernel selection and launch.
// The exported functions are declared and documented in include/qgemm.h.
#include "../../include/qgemm.h"

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "w4a16.cuh"
#include "w4a16_decode.cuh"
#include "w4a16_gs.cuh"
#include "w4a16_wide.cuh"
#include "act_quant.cuh"
#include "w4a8.cuh"
#include "w8a8.cuh"
#include "w8a8_rows.cuh"

namespace {

thread_local char g_err[512] = "";
unsigned long long g_wait_limit_ns = 2000ull * 1000ull * 1000ull;

int fail(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return -1;
}

#define CUDA_OK(expr)                                                                      \
  do {                                                                                     \
    cudaError_t e_ = (expr);                                                               \
    if (e_ != cudaSuccess) return fail("%s failed: %s", #expr, cudaGetErrorString(e_));   \
  } while (0)

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

constexpr int kMaxDevices = 64;
struct DeviceState {
  std::atomic<bool> ready{false};
  int sm_count = 0;
};
std::mutex g_mu;
DeviceState g_dev[kMaxDevices];
EncodeTiledFn g_encode = nullptr;

// Kernels that are to be resident beside one another - a GEMM kernel and the next call's pre-pass - want all of an SM's memory that
// can be as shared memory.  The driver by itself takes as little as one of them needs, 196 KB for the 187 of the 16-token group-sum
// kernel, beside which the pre-pass's 21 KB found no room: 8 x 16 x 4096 x 4096, call after call, 22.0 us instead of 18.6, 27 x 15 x
// 1024 x 3120 17.0 / 14.8, W4A8 27 x 3328 x 2320 20.3 / 18.1, 64 x 4096 x 14336 23.7 / 22.0 (as one graph it mostly did find room).
// A kernel by itself is the slower for the smaller cache: 16 x 4096 x 4096 in a single launch 8.46, 8.37 with 196 KB.
template <typename K>
int most_shared_memory(K kernel) {
  CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  return 0;
}
template <typename K>
int set_smem(K kernel, int bytes, bool beside_pre_pass = false) {
  CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return beside_pre_pass ? most_shared_memory(kernel) : 0;
}

template <int BN>
int set_smem_w8() {
  using C = qg::W8Cfg<BN>;
  if (set_smem(qg::w8a8_gemm_kernel<BN, false, false>, C::SMEM_BYTES)) return -1;
  if (set_smem(qg::w8a8_gemm_kernel<BN, false, true>, C::SMEM_BYTES)) return -1;
  if (set_smem(qg::w8a8_gemm_kernel<BN, true, false>, C::SMEM_BYTES)) return -1;
  if (set_smem(qg::w8a8_gemm_kernel<BN, true, true>, C::SMEM_BYTES)) return -1;
  if constexpr (BN == 256) {  // the forms of two CTAs
    if (set_smem(qg::w8a8_gemm_kernel<256, false, false, qg::W8_SPLITK>, C::SMEM_BYTES)) return -1;
    if (set_smem(qg::w8a8_gemm_kernel<256, false, true, qg::W8_SPLITK>, C::SMEM_BYTES)) return -1;
    constexpr int pair_bytes = qg::W8Cfg<256, qg::W8_PAIR>::SMEM_BYTES;
    if (set_smem(qg::w8a8_gemm_kernel<256, false, false, qg::W8_PAIR>, pair_bytes)) return -1;
    if (set_smem(qg::w8a8_gemm_kernel<256, false, true, qg::W8_PAIR>, pair_bytes)) return -1;
    if (set_smem(qg::w8a8_gemm_kernel<256, true, false, qg::W8_PAIR>, pair_bytes)) return -1;
    if (set_smem(qg::w8a8_gemm_kernel<256, true, true, qg::W8_PAIR>, pair_bytes)) return -1;
  }
  return 0;
}
template <int FLUSH>
int set_smem_w4d() {
  if (set_smem(qg::w4a16_decode_kernel<FLUSH, 1, false>, qg::W4DCfg<1>::SMEM_BYTES)) return -1;
  if (set_smem(qg::w4a16_decode_kernel<FLUSH, 1, true>, qg::W4DCfg<1>::SMEM_BYTES)) return -1;
  if (set_smem(qg::w4a16_decode_kernel<FLUSH, 2, false>, qg::W4DCfg<2>::SMEM_BYTES)) return -1;
  if (set_smem(qg::w4a16_decode_kernel<FLUSH, 2, true>, qg::W4DCfg<2>::SMEM_BYTES)) return -1;
  return 0;
}
template <int MT>
int set_smem_w4i8() {
  using C = qg::W4I8Cfg<MT>;
  if (set_smem(qg::w4a8_gemm_kernel<MT, false>, C::SMEM_BYTES, true)) return -1;
  if (set_smem(qg::w4a8_gemm_kernel<MT, true>, C::SMEM_BYTES, true)) return -1;
  if constexpr (MT == 16) {
    if (set_smem(qg::w4a8_gemm_kernel<MT, false, true>, C::SMEM_BYTES, true)) return -1;
    if (set_smem(qg::w4a8_gemm_kernel<MT, true, true>, C::SMEM_BYTES, true)) return -1;
  }
  return 0;
}
template <int MT>
int set_smem_w4() {
  using C = qg::W4Cfg<MT>;
  if (set_smem(qg::w4a16_gemm_kernel<MT, false>, C::SMEM_BYTES)) return -1;
  if (set_smem(qg::w4a16_gemm_kernel<MT, true>, C::SMEM_BYTES)) return -1;
  return 0;
}

template <int MT>
int set_smem_w4g() {
  using C = qg::W4GCfg<MT>;
  constexpr int zt_bytes = qg::W4GCfg<MT, true>::SMEM_BYTES;
  if (set_smem(qg::w4a16_gs_kernel<MT, false>, C::SMEM_BYTES, true)) return -1;
  if (set_smem(qg::w4a16_gs_kernel<MT, true>, C::SMEM_BYTES, true)) return -1;
  if (set_smem(qg::w4a16_gs_kernel<MT, false, true>, C::SMEM_BYTES, true)) return -1;
  if (set_smem(qg::w4a16_gs_kernel<MT, true, true>, C::SMEM_BYTES, true)) return -1;
  if (set_smem(qg::w4a16_gs_kernel<MT, false, false, true>, zt_bytes, true)) return -1;
  if (set_smem(qg::w4a16_gs_kernel<MT, true, false, true>, zt_bytes, true)) return -1;
  if constexpr (MT == 16) {
    if (set_smem(qg::w4a16_gs_kernel<16, false, false, false, true>, C::SMEM_BYTES)) return -1;
    if (set_smem(qg::w4a16_gs_kernel<16, true, false, false, true>, C::SMEM_BYTES)) return -1;
  }
  return 0;
}

int set_smem_w8r() {
  constexpr int smem = qg::W8R_RING_BYTES_ONE + qg::W8R_EXTRA_BYTES;
  if (set_smem(qg::w8a8_rows_kernel<false, false>, smem)) return -1;
  if (set_smem(qg::w8a8_rows_kernel<false, true>, smem)) return -1;
  if (set_smem(qg::w8a8_rows_kernel<true, false>, smem)) return -1;
  return set_smem(qg::w8a8_rows_kernel<true, true>, smem);
}
template <bool PAIR>
int set_smem_w4w() {
  if (set_smem(qg::w4a16_wide_kernel<false, false, PAIR>, qg::W4WideCfg<false>::SMEM_BYTES)) return -1;
  if (set_smem(qg::w4a16_wide_kernel<true, false, PAIR>, qg::W4WideCfg<false>::SMEM_BYTES)) return -1;
  if (set_smem(qg::w4a16_wide_kernel<false, true, PAIR>, qg::W4WideCfg<true>::SMEM_BYTES)) return -1;
  return set_smem(qg::w4a16_wide_kernel<true, true, PAIR>, qg::W4WideCfg<true>::SMEM_BYTES);
}

// The set-up of the current device, once per device.
int ensure_device(int* sm_count) {
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail("device index %d out of range", dev);
  DeviceState& st = g_dev[dev];
  if (st.ready.load(std::memory_order_acquire)) {  // every call but the first one per device
    *sm_count = st.sm_count;
    return 0;
  }
  std::lock_guard<std::mutex> lock(g_mu);
  if (!st.ready.load(std::memory_order_relaxed)) {
    cudaDeviceProp prop;
    CUDA_OK(cudaGetDeviceProperties(&prop, dev));
    if (prop.major != 10) return fail("libqgemm needs an sm_100a device (B200); device %d is sm_%d%d", dev, prop.major, prop.minor);
    if (g_encode == nullptr) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qres;
      CUDA_OK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
      if (qres != cudaDriverEntryPointSuccess || fn == nullptr) return fail("cuTensorMapEncodeTiled not available from the driver");
      g_encode = reinterpret_cast<EncodeTiledFn>(fn);
    }
    if (set_smem_w8<128>() || set_smem_w8<256>()) return -1;
    if (set_smem_w4<16>()) return -1;
    if (set_smem_w4g<16>() || set_smem_w4g<32>() || set_smem_w4g<64>()) return -1;
    if (set_smem_w4i8<16>() || set_smem_w4i8<32>() || set_smem_w4i8<64>() || set_smem_w4i8<128>()) return -1;
    if (set_smem_w8r() || set_smem_w4w<false>() || set_smem_w4w<true>()) return -1;
    if (most_shared_memory(qg::w4g_prepare_activations<false>) || most_shared_memory(qg::w4g_prepare_activations<true>)) return -1;
    if (most_shared_memory(qg::w4a8_prepare_activations<12>) || most_shared_memory(qg::w4a8_prepare_activations<16>)) return -1;
    if (most_shared_memory(qg::w4a8_quant_prepare_activations<12>) || most_shared_memory(qg::w4a8_quant_prepare_activations<16>)) return -1;
    if (set_smem_w4d<0>() || set_smem_w4d<1>() || set_smem_w4d<2>() || set_smem_w4d<4>()) return -1;
    st.sm_count = prop.multiProcessorCount;
    st.ready.store(true, std::memory_order_release);
  }
  *sm_count = st.sm_count;
  return 0;
}

// rank-2/3 row-major tensor map; dims/box innermost first; strides in bytes for dims 1.. (innermost is dense).
int encode_map(CUtensorMap* map, CUtensorMapDataType dt, int rank, const void* base, const uint64_t* dims,
               const uint64_t* strides_bytes, const uint32_t* box, CUtensorMapSwizzle swz) {
  cuuint64_t gdim[3], gstr[2];
  cuuint32_t bx[3], es[3];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i > 0) gstr[i - 1] = strides_bytes[i - 1];
  }
  CUresult r = g_encode(map, dt, (cuuint32_t)rank, const_cast<void*>(base), gdim, gstr, bx, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
  return 0;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Launch `kernel` so that it may start while the kernel in front of it on the stream is still running
// (programmatic dependent launch); the kernel itself waits before it reads that kernel's results.
// QGEMM_PDL=0 falls back to plain stream order.
template <typename... KArgs, typename... Args>
int launch_pdl(void (*kernel)(KArgs...), int grid, int threads, int smem, cudaStream_t s, Args&&... args) {
  static const int pdl = getenv("QGEMM_PDL") ? atoi(getenv("QGEMM_PDL")) : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
  return 0;
}

// Rasterisation band: the tiles of `group_m` consecutive row blocks are walked column block by column block, so a
// wave of CTAs shares few B tiles and the band's A rows (group_m x 128 x K bytes) stay in L2 while every B tile
// streams through once per band.  As many row blocks as keep the band's A rows within 34 MB, at least 8: config 3
// takes all 32 row blocks (16.8 MB, B read from DRAM once instead of four times: 172 -> 165 us; 16 or 24 row blocks:
// 170 us).
// Grouped form (groups > 0): 8 while L2 keeps a group's B beside the band's A.  A higher band holds row blocks of several groups,
// whose B tiles do not share anything, and comes back to its A rows only after all of those.  A B that L2 does not keep streams
// through once per band: then all row blocks that a group has in the mean, within the 34 MB.  us, in turn, bands of 8 / of a
// group's row blocks / of 34 MB: 16 groups, 8192 x 7168 x 2048 95.9 / 95.9 / 100.4 (of 32 row blocks); 4 groups, 8192 x 2048 x 4096
// 55.2 / 56.2 / 57.7; one group, 4096 x 7168 x 4096 (29 MB of B) 85.1 / 87.1; 8192 x 4096 x 8192 (34 MB) 187.5 / 184.7, two groups
// 189.2 / 188.3; 4096 x 7168 x 7168 (51 MB) 149.0 / 143.5; 8192 x 4096 x 14336 (59 MB), one group 337 / 324, two 338 / 328 / 328,
// four 341 / 334 / 337, eight 345 / 345 / 354.
int w8_group_m(int64_t m_tiles, int64_t k_bytes, int64_t groups, int64_t b_bytes) {
  static const int forced = getenv("QGEMM_W8_GROUP_M") ? atoi(getenv("QGEMM_W8_GROUP_M")) : 0;  // tuning override
  int64_t g = (34ll << 20) / (128 * (k_bytes > 0 ? k_bytes : 1));
  if (groups > 0) g = b_bytes <= (40ll << 20) ? 8 : std::min(g, m_tiles / groups);
  if (forced > 0) g = forced;
  if (g < 8) g = 8;
  if (g > m_tiles) g = m_tiles;
  return (int)(g > 0 ? g : 1);
}

template <int BN, bool NK, bool BF>
int launch_w8(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const qg::W8A8Params& p, int grid,
              cudaStream_t s) {
  return launch_pdl(qg::w8a8_gemm_kernel<BN, NK, BF>, grid, qg::W8_THREADS, qg::W8Cfg<BN>::SMEM_BYTES, s, tmA, tmB, tmC, p);
}

// The forms in which a cluster of two CTAs makes a tile: `clusters` of them.
template <bool NK, bool BF, qg::W8Form FORM>
int launch_w8_clusters(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmC, const qg::W8A8Params& p,
                       int clusters, cudaStream_t s) {
  static const int pdl = getenv("QGEMM_PDL") ? atoi(getenv("QGEMM_PDL")) : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * clusters));
  cfg.blockDim = dim3((unsigned)qg::W8_THREADS);
  cfg.dynamicSmemBytes = (size_t)qg::W8Cfg<256, FORM>::SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  CUDA_OK(cudaLaunchKernelEx(&cfg, qg::w8a8_gemm_kernel<256, NK, BF, FORM>, tmA, tmB, tmC, p));
  return 0;
}
// Few-token form: clusters of S CTAs, a programmatic dependent of whatever is in front of it on the stream.
template <bool NK, bool BF>
int launch_w8_rows(const CUtensorMap& tmA, const CUtensorMap& tmB, const qg::W8RowsParams& p, int grid, int S, cudaStream_t s) {
  static const int pdl = getenv("QGEMM_PDL") ? atoi(getenv("QGEMM_PDL")) : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(qg::W8R_THREADS);
  cfg.dynamicSmemBytes = (size_t)(p.ring + qg::W8R_EXTRA_BYTES);
  cfg.stream = s;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  CUDA_OK(cudaLaunchKernelEx(&cfg, qg::w8a8_rows_kernel<NK, BF>, tmA, tmB, p));
  return 0;
}

int launch_w4(bool bf, const CUtensorMap& tmW, const CUtensorMap& tmS, const CUtensorMap& tmA,
              const qg::W4A16Params& p, int grid, cudaStream_t s) {
  if (bf) return launch_pdl(qg::w4a16_gemm_kernel<16, true>, grid, qg::W4_THREADS, qg::W4Cfg<16>::SMEM_BYTES, s, tmW, tmS, tmA, p);
  return launch_pdl(qg::w4a16_gemm_kernel<16, false>, grid, qg::W4_THREADS, qg::W4Cfg<16>::SMEM_BYTES, s, tmW, tmS, tmA, p);
}
constexpr int64_t kW4MaxGrid = 1024;
constexpr int64_t kW4CounterBytes = kW4MaxGrid * 4;

// Test hook (qgemm_debug_withhold_commit): see W4GDebug, and `withhold` of W8A8Params and W4A16Params.
int g_withhold = 0;

// `tmZ` non-null: the zeros-tensor instantiation (not combined with the gathered form).
template <int MT>
int launch_w4g(bool bf, const CUtensorMap& tmW, const CUtensorMap& tmS, const CUtensorMap* tmZ, const CUtensorMap& tmA,
               const qg::W4A16Params& p, int grid, cudaStream_t s) {
  qg::W4GDebug dbg;
  dbg.withhold_last_commit = g_withhold;
  constexpr int smem = qg::W4GCfg<MT>::SMEM_BYTES, smem_zt = qg::W4GCfg<MT, true>::SMEM_BYTES;
  if (tmZ != nullptr) {
    if (bf) return launch_pdl(qg::w4a16_gs_kernel<MT, true, false, true>, grid, qg::W4G_THREADS, smem_zt, s, tmW, tmS, *tmZ, tmA, p, dbg);
    return launch_pdl(qg::w4a16_gs_kernel<MT, false, false, true>, grid, qg::W4G_THREADS, smem_zt, s, tmW, tmS, *tmZ, tmA, p, dbg);
  }
  if (p.n_dst > 0) {
    if (bf) return launch_pdl(qg::w4a16_gs_kernel<MT, true, true>, grid, qg::W4G_THREADS, smem, s, tmW, tmS, tmS, tmA, p, dbg);
    return launch_pdl(qg::w4a16_gs_kernel<MT, false, true>, grid, qg::W4G_THREADS, smem, s, tmW, tmS, tmS, tmA, p, dbg);
  }
  if (bf) return launch_pdl(qg::w4a16_gs_kernel<MT, true>, grid, qg::W4G_THREADS, smem, s, tmW, tmS, tmS, tmA, p, dbg);
  return launch_pdl(qg::w4a16_gs_kernel<MT, false>, grid, qg::W4G_THREADS, smem, s, tmW, tmS, tmS, tmA, p, dbg);
}

// The wide tiles, `workers` CTAs or pairs of them; a programmatic dependent of the pre-pass.
template <bool BF, bool ZT, bool PAIR>
int launch_w4w(const CUtensorMap& tmW, const CUtensorMap& tmS, const CUtensorMap& tmZ, const CUtensorMap& tmA,
               const qg::W4A16Params& p, int mt, int zero_mode, int workers, cudaStream_t s) {
  static const int pdl = getenv("QGEMM_PDL") ? atoi(getenv("QGEMM_PDL")) : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(PAIR ? 2 * workers : workers));
  cfg.blockDim = dim3((unsigned)qg::W4W_THREADS);
  cfg.dynamicSmemBytes = (size_t)qg::W4WideCfg<ZT>::SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PAIR ? 2 : 1;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  CUDA_OK(cudaLaunchKernelEx(&cfg, qg::w4a16_wide_kernel<BF, ZT, PAIR>, tmW, tmS, tmZ, tmA, p, mt, zero_mode));
  return 0;
}
template <bool PAIR>
int launch_w4w(bool bf, bool zt, const CUtensorMap& tmW, const CUtensorMap& tmS, const CUtensorMap& tmZ, const CUtensorMap& tmA,
               const qg::W4A16Params& p, int mt, int zero_mode, int workers, cudaStream_t s) {
  if (zt) return bf ? launch_w4w<true, true, PAIR>(tmW, tmS, tmZ, tmA, p, mt, zero_mode, workers, s) : launch_w4w<false, true, PAIR>(tmW, tmS, tmZ, tmA, p, mt, zero_mode, workers, s);
  return bf ? launch_w4w<true, false, PAIR>(tmW, tmS, tmZ, tmA, p, mt, 0, workers, s) : launch_w4w<false, false, PAIR>(tmW, tmS, tmZ, tmA, p, mt, 0, workers, s);
}

// The pre-pass of the group-sum kernel.
int launch_w4g_prepare(const void* A, void* out, const qg::W4A16Params& p, bool is_bf16, int sms, cudaStream_t s) {
  constexpr int warps = qg::W4G_PREP_THREADS / 32;
  const long long rows = (long long)p.batch * p.M, slabs = rows * p.KS;
  if (slabs > 0x3fffffffll) return fail("qgemm_w4a16: activation tensor too large");
  // A block per SM at most, so that all are resident early, and each warp's share in equal rounds.  Above four rounds throughput
  // counts for more than an early start: a block for every round.  Ten of them are resident on an SM (20 KB of shared memory and 1 KB
  // beside it each), but with no more than ten launched warps of the last round come to a second one.  us, one block per SM / a block
  // for every round (one for every 128 chunks of 32 k, before): 24 x 60 x 7424 x 1408 51.9 / 46.4 (51.0), 32 x 64 x 8192 x 1024 63.6 /
  // 52.7 (58.7; ten per SM 54.6), 40 x 64 x 8192 x 1024 - / 65.6 (72.6; ten per SM 67.0, eleven 67.0); from two rounds on 20 x 48 x 4096
  // x 2048 33.9 / 35.8 (37.0), 8 x 64 x 8192 x 1024 25.4 / 27.5 (28.0), but 24 x 64 x 4096 x 4096 70.3 / 69.0.
  const long long each = (slabs + warps * sms - 1) / (warps * sms), rounds = (each + qg::W4G_PREP_LANDING - 1) / qg::W4G_PREP_LANDING;
  const int per = (int)((each + rounds - 1) / rounds);
  const long long blocks = (slabs + warps * per - 1) / (warps * per);
  const int grid = (int)(rounds > 4 ? blocks : std::min<long long>(sms, blocks));
  auto kernel = per <= qg::W4G_PREP_REGS ? qg::w4g_prepare_activations<false> : qg::w4g_prepare_activations<true>;
  return launch_pdl(kernel, grid, qg::W4G_PREP_THREADS, 0, s, static_cast<const uint4*>(A), static_cast<uint8_t*>(out), (int)rows, p.M,
                    p.K, p.KS, is_bf16 ? 1 : 0, per, reinterpret_cast<uint4*>(p.ws_counters), (int)(kW4CounterBytes / 4));
}

// Single-launch form of the group-sum kernel (see its SMALL parameter): clusters of `cluster` CTAs, one tile per cluster,
// no pre-pass in front.  Still a programmatic dependent of whatever is in front of it on the stream.
int launch_w4g_small(bool bf, const CUtensorMap& tmW, const CUtensorMap& tmS, const qg::W4A16Params& p, int grid, int cluster, cudaStream_t s) {
  static const int pdl = getenv("QGEMM_PDL") ? atoi(getenv("QGEMM_PDL")) : 1;
  qg::W4GDebug dbg;
  dbg.withhold_last_commit = g_withhold;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)qg::W4G_THREADS);
  cfg.dynamicSmemBytes = (size_t)qg::W4GCfg<16>::SMEM_BYTES;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  if (bf) CUDA_OK(cudaLaunchKernelEx(&cfg, qg::w4a16_gs_kernel<16, true, false, false, true>, tmW, tmS, tmS, tmS, p, dbg));
  else CUDA_OK(cudaLaunchKernelEx(&cfg, qg::w4a16_gs_kernel<16, false, false, false, true>, tmW, tmS, tmS, tmS, p, dbg));
  return 0;
}

// The group-sum kernel (w4a16_gs.cuh) serves up to 64 tokens when the scale groups are 128 wide, a multiple of
// 256 or the whole K (or there are no scales); it is faster than the register-operand decode kernel at every
// token count (K=8192, N=28672: 25 against 40 us at one token).  Groups of 32 / 64: see w4_route.  QGEMM_W4_GS=0 disables
// the group-sum kernel, QGEMM_W4_GS_MIN_M raises the token count from which it is used.
int w4_gs_min_m() {
  static const int v = getenv("QGEMM_W4_GS_MIN_M") ? atoi(getenv("QGEMM_W4_GS_MIN_M")) : 1;
  return v;
}
bool w4_gs_shape_ok(int64_t M, bool has_scales, int64_t group, int64_t K) {
  static const int enabled = getenv("QGEMM_W4_GS") ? atoi(getenv("QGEMM_W4_GS")) : 1;
  if (!enabled || M > 64 || M < w4_gs_min_m()) return false;
  return !has_scales || group == 128 || group % 256 == 0 || group >= K;
}

template <int FLUSH, int NB>
int launch_w4d_nb(bool bf, const CUtensorMap& tmW, const CUtensorMap& tmS, const CUtensorMap& tmA,
                  const qg::W4A16Params& p, int grid, cudaStream_t s) {
  if (bf) return launch_pdl(qg::w4a16_decode_kernel<FLUSH, NB, true>, grid, qg::W4D_THREADS, qg::W4DCfg<NB>::SMEM_BYTES, s, tmW, tmS, tmA, p);
  return launch_pdl(qg::w4a16_decode_kernel<FLUSH, NB, false>, grid, qg::W4D_THREADS, qg::W4DCfg<NB>::SMEM_BYTES, s, tmW, tmS, tmA, p);
}
template <int FLUSH>
int launch_w4d(bool bf, int mt, const CUtensorMap& tmW, const CUtensorMap& tmS, const CUtensorMap& tmA,
               const qg::W4A16Params& p, int grid, cudaStream_t s) {
  if (mt == 16) return launch_w4d_nb<FLUSH, 2>(bf, tmW, tmS, tmA, p, grid, s);
  return launch_w4d_nb<FLUSH, 1>(bf, tmW, tmS, tmA, p, grid, s);
}
// Narrow scale groups: token counts up to this use the register-operand streaming kernel (w4a16_decode.cuh), above it
// the tcgen05 kernel (w4a16.cuh).
int w4_decode_max_m() {
  static int v = -1;
  if (v < 0) {
    v = 8;
    if (const char* e = getenv("QGEMM_W4_DECODE_MAX_M")) v = atoi(e) < 16 ? atoi(e) : 16;
  }
  return v;
}
bool w4_use_decode(int64_t M) { return M <= w4_decode_max_m(); }
// Token-tile height: 16, 32 or 64 for the group-sum kernel, 8 or 16 for the decode kernel, 16 for w4a16.cuh's.
int w4_pick_mt(int64_t M, bool gs) {
  if (gs) return M <= 16 ? 16 : (M <= 32 ? 32 : 64);
  return w4_use_decode(M) && M <= 8 ? 8 : 16;
}

__global__ void unpack_int4_kernel(const uint8_t* __restrict__ packed, int8_t* __restrict__ out, long long n_bytes,
                                   int signed_nibbles) {
  // 16 packed bytes -> 32 int8 values per thread; low nibble first.
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long base = i * 16;
  if (base >= n_bytes) return;
  if (base + 16 <= n_bytes) {
    const uint4 v = *reinterpret_cast<const uint4*>(packed + base);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t lo = w[j] & 0x0f0f0f0fu;         // even elements
      uint32_t hi = (w[j] >> 4) & 0x0f0f0f0fu;  // odd elements
      if (signed_nibbles) {                     // two's complement nibble: (x ^ 8) - 8 per byte
        lo = __vsub4(lo ^ 0x08080808u, 0x08080808u);
        hi = __vsub4(hi ^ 0x08080808u, 0x08080808u);
      }
      o[2 * j] = __byte_perm(lo, hi, 0x5140);      // e0 o0 e1 o1
      o[2 * j + 1] = __byte_perm(lo, hi, 0x7362);  // e2 o2 e3 o3
    }
    uint4* dst = reinterpret_cast<uint4*>(out + base * 2);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
  } else {
    for (long long b = base; b < n_bytes; ++b) {
      int lo = packed[b] & 0xF, hi = packed[b] >> 4;
      if (signed_nibbles) {
        lo = (lo ^ 8) - 8;
        hi = (hi ^ 8) - 8;
      }
      out[2 * b] = (int8_t)lo;
      out[2 * b + 1] = (int8_t)hi;
    }
  }
}

}  // namespace

template <int MT>
static int launch_w4i8(bool sgn, const CUtensorMap& tmW, const CUtensorMap& tmA, const qg::W4A8Params& p, int grid,
                       cudaStream_t s) {
  if constexpr (MT == 16) {
    if (p.dp_rounds > 0 && p.KS >= 24) {
      if (sgn) return launch_pdl(qg::w4a8_gemm_kernel<MT, true, true>, grid, qg::W4I8Cfg<MT>::THREADS, qg::W4I8Cfg<MT>::SMEM_BYTES, s, tmW, tmA, p);
      return launch_pdl(qg::w4a8_gemm_kernel<MT, false, true>, grid, qg::W4I8Cfg<MT>::THREADS, qg::W4I8Cfg<MT>::SMEM_BYTES, s, tmW, tmA, p);
    }
  }
  if (sgn) return launch_pdl(qg::w4a8_gemm_kernel<MT, true>, grid, qg::W4I8Cfg<MT>::THREADS, qg::W4I8Cfg<MT>::SMEM_BYTES, s, tmW, tmA, p);
  return launch_pdl(qg::w4a8_gemm_kernel<MT, false>, grid, qg::W4I8Cfg<MT>::THREADS, qg::W4I8Cfg<MT>::SMEM_BYTES, s, tmW, tmA, p);
}

// Fused path of qgemm_w4a8 for up to 128 tokens: no int8 copy of the weights; the caller's [N, K] workspace
// only holds the small scratch (arrival counters, int32 partial sums, reordered activations, row sums).
// Returns 1 when the problem does not qualify (the caller then takes the two-kernel path).
// `A` int8 [M, K]; or, with `X` non-null, bf16 / f16 activations that the pre-pass quantises per token itself
// (scales to `scale_out`).
static int w4a8_fused(const int8_t* A, const uint8_t* qB, int8_t* workspace, int* C, int64_t M, int64_t N, int64_t K,
                      int signed_nibbles, uint32_t* status, cudaStream_t s, const void* X = nullptr, int x_is_bf16 = 0,
                      int round_scale = 0, float* scale_out = nullptr) {
  static const int enabled = getenv("QGEMM_W4A8_FUSED") ? atoi(getenv("QGEMM_W4A8_FUSED")) : 1;
  if (!enabled || M > 128 || !aligned16(workspace)) return 1;
  int sms = 0;
  if (ensure_device(&sms)) return -1;
  const int mt = M <= 16 ? 16 : (M <= 32 ? 32 : (M <= 64 ? 64 : 128));
  const int64_t grid_max = sms < kW4MaxGrid ? sms : kW4MaxGrid;
  const int64_t partial_bytes = grid_max * 2 * (int64_t)mt * 128 * 4;
  const int64_t a_bytes = ((M * K + 255) / 256) * 256;
  const int64_t need = kW4CounterBytes + partial_bytes + a_bytes + ((M * 4 + 255) / 256) * 256;
  if (need > N * K) return 1;  // the caller's workspace is [N, K] int8
  uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
  uint8_t* a_prepared = ws + kW4CounterBytes + partial_bytes;
  // Blocks of the pre-pass per row: as many as leave one block for every SM, four above 64 tokens, where they do not fit beside a CTA
  // of the GEMM kernel; one for up to four rows, whose few blocks delay nobody (2 x 6144 x 1824 13.6 us, 14.7 with eight, 3 x 4096 x
  // 14336 12.9 / 14.3).  The sums over their parts of K stand behind the counters that are used.
  const int parts = (int)std::max<int64_t>(1, std::min<int64_t>({M <= 4 ? 1 : qg::W4I8_PREP_MAX_PARTS, M <= 64 ? sms / M : 4 * sms / M, (kW4MaxGrid - grid_max) / M}));
  int* row_sums = parts > 1 ? reinterpret_cast<int*>(ws) + grid_max : reinterpret_cast<int*>(a_prepared + a_bytes);

  CUtensorMap tmW, tmA;
  {
    const uint64_t dims[2] = {(uint64_t)(K / 2), (uint64_t)N};
    const uint64_t str[1] = {(uint64_t)(K / 2)};
    const uint32_t box[2] = {128, 128};
    if (encode_map(&tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, qB, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }
  {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    const uint64_t str[1] = {(uint64_t)K};
    const uint32_t box[2] = {128, (uint32_t)mt};
    if (encode_map(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, a_prepared, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }
  qg::W4A8Params p;
  p.C = C;
  p.ws_counters = reinterpret_cast<uint32_t*>(ws);
  p.ws_partials = reinterpret_cast<int*>(ws + kW4CounterBytes);
  p.row_sums = row_sums;
  p.row_parts = parts;
  p.M = (int)M;
  p.N = (int)N;
  p.K = (int)K;
  p.n_tiles = (int)((N + 127) / 128);
  p.KS = (int)((K + 255) / 256);
  p.status = status;
  p.wait_limit_ns = g_wait_limit_ns;
  const int64_t items = (int64_t)p.n_tiles * p.KS, grid = grid_max < items ? grid_max : items;
  // As the group-sum kernel: whole tiles where there are enough, the remainder (with one whole round, when it is small) cut.
  const int64_t rounds = p.n_tiles / grid, left = p.n_tiles % grid;
  const bool borrow = rounds != 0 && left != 0 && 2 * left < grid;
  p.dp_rounds = (int)(borrow ? rounds - 1 : rounds);
  p.sk_tiles = (int)(borrow ? left + grid : left);
  // a programmatic dependent of whatever is in front: behind another call of this operator it is resident early
  if (X != nullptr) {
    auto prepare = M <= 16 ? qg::w4a8_quant_prepare_activations<12> : qg::w4a8_quant_prepare_activations<16>;
    const int kept = 16 * (int)std::min<int64_t>(K / 8, qg::W4I8_PREP_KEPT);
    if (launch_pdl(prepare, (int)M * parts, qg::W4I8_PREP_THREADS, kept, s, static_cast<const uint4*>(X), x_is_bf16, round_scale,
                   reinterpret_cast<uint2*>(a_prepared), row_sums, scale_out, p.ws_counters, (int)grid_max, (int)K, (int)M, parts))
      return -1;
  } else if (launch_pdl(M <= 16 ? qg::w4a8_prepare_activations<12> : qg::w4a8_prepare_activations<16>, (int)M * parts,
                        qg::W4I8_PREP_THREADS, 0, s, reinterpret_cast<const uint2*>(A), reinterpret_cast<uint2*>(a_prepared), row_sums, p.ws_counters,
                        (int)grid_max, (int)K, (int)M, parts))
    return -1;
  const bool sgn = signed_nibbles != 0;
  switch (mt) {
    case 16: return launch_w4i8<16>(sgn, tmW, tmA, p, (int)grid, s);
    case 32: return launch_w4i8<32>(sgn, tmW, tmA, p, (int)grid, s);
    case 64: return launch_w4i8<64>(sgn, tmW, tmA, p, (int)grid, s);
    default: return launch_w4i8<128>(sgn, tmW, tmA, p, (int)grid, s);
  }
}

extern "C" {

int qgemm_version(void) { return 1006; }  // 1.6: + in-flight zero tensors, W4A8 with the activation quantiser fused into its pre-pass

const char* qgemm_last_error(void) { return g_err; }

void qgemm_set_wait_limit_ms(uint32_t ms) { g_wait_limit_ns = (unsigned long long)ms * 1000000ull; }

void qgemm_debug_withhold_commit(int on) { g_withhold = on >= 2 && on <= 4 ? on : (on ? 1 : 0); }

int qgemm_init(void) {
  int sms = 0;
  return ensure_device(&sms);
}

// How the few-token form (w8a8_rows.cuh) takes `tiles` tiles: over how many CTAs it cuts their K, and the bytes of a CTA's pipeline.
// split 0: w8a8.cuh is the faster one.
// The cut.  One CTA per SM, as long as it saves each CTA four k blocks; clusters of eight from 32 k blocks on, as long as each CTA of
// theirs finds an SM of its own: 15 of them did on the chip this was measured on, and one is left as a margin.  us, cut in four / in
// eight, 8, 32 and 128 tokens: 1792 columns (14 clusters), K = 4096 5.32 / 5.41, 6.20 / 5.67, 7.64 / 7.57, K = 8192 7.74 / 7.31, 9.09 /
// 7.36, 10.00 / 9.95 ([N, K] weights 5.26 / 5.28, 5.84 / 5.41, 7.75 / 7.37, 7.59 / 7.36, 8.12 / 7.51, 10.27 / 9.84); 2048 columns (16),
// K = 4096 5.50 / 7.03, 6.15 / 7.06, 7.86 / 9.75.  A second CTA per SM by a further cut does not pay.
// The pipeline.  96 KB, beside which the next call's CTA finds room, where that holds a CTA's whole K (64 tiles of K = 1024, cut in two,
// 96 / 208 KB: 17 tokens 4.54 / 4.87 us, 40 tokens 6.3 / 6.5), for up to 16 tokens of [K, N] weights, and where CTAs share SMs; else 208
// KB.  us, calls one after another: [K, N] 16 x 8192 x 8192 14.2 / 14.8, 16 x 4096 x 14336 12.6 / 12.8, 17 x 4096 x 14336 14.5 / 13.5, 32 x
// 2048 x 14336 9.4 / 8.7, 32 x 1024 x 14336 6.7 / 6.6, [N, K] 16 x 8192 x 8192 15.0 / 14.9, 32 x 8192 x 8192 16.7 / 15.0, 8 x 1024 x 14336 5.9 /
// 5.9, 8 x 1536 x 12288 6.9 / 6.8.  ([K, N], 110 shapes: at 4, 12 and 16 tokens 208 KB is 2 % slower in the mean, 3 % above eight blocks a
// CTA; at 17 .. 32 tokens 1 and 3 % faster.)
// Clusters of four do not fill all SMs with one CTA each either, 132 of 148 on that chip, 128 on another: 24 fewer (57 x 1824 x 4240, 34
// clusters, 10.3 us with 208 KB, 7.0 with 96).
// The choice.  Per tile this form pays for its tokens and saves the k blocks that other CTAs take: up to 48 tokens always, above that
// when the cut saves three blocks, and one more for every eight tokens, up to 64 also uncut from eleven blocks on.  (220 shapes of
// 41 .. 128 tokens per tile: 0.5 % behind the better one in the mean.)  The time by w8a8.cuh over this form's: 124 tokens, 188 tiles,
// K = 4608 0.64; 54 tokens, 73 tiles, K = 640 0.96; 60 tokens, 112 tiles, K = 2048 1.16; 109 tokens, 5 tiles cut in four, K = 1920 1.04.
// From 150 shapes (1 .. 10 problems of 1 .. 512 tokens, K 512 .. 8192, N 512 .. 14336, weights from DRAM; every cut, both pipelines and
// the other kernel in turn): 1.0 % behind the best in the mean, where the rule before (two CTAs per SM from eight blocks each on, 96 KB)
// was 4.1 %.  us, before / after: 24 x 4096 x 14336 14.7 / 13.6, 128 x 8192 x 8192 20.7 / 18.5, 71 tokens of 140 tiles, K = 4864 17.5 /
// 15.3, 24 x 8192 x 4096 12.1 / 11.1, 13 x 512 x 3008 4.2 / 3.6; 256 x 1024 x 1024 6.4 by this form, 5.9 by w8a8.cuh.
struct W8RowsPlan {
  int split, ring;
};
static W8RowsPlan w8_rows_plan(int64_t tiles, int64_t k_blocks, int64_t tokens, bool kn, int64_t sms) {
  auto saved = [&](int64_t n) { return k_blocks - (k_blocks + n - 1) / n; };
  int64_t S = 1;
  if (2 * tiles <= sms && saved(2) >= 4) S = 2;
  if (4 * tiles <= sms && saved(4) >= 4) S = 4;
  if (8 * tiles <= sms - 36 && k_blocks >= 32) S = 8;
  static_assert(qg::W8R_MAX_SPLIT == 8, "cuts above");
  const bool alone = S < 4 ? S * tiles <= sms : (S == 4 && S * tiles <= sms - 24);
  const bool held = (k_blocks + S - 1) / S * (qg::W8R_W_BYTES + 128 * tokens) <= qg::W8R_RING_BYTES;
  const W8RowsPlan plan{(int)S, alone && !held && (!kn || tokens > 16) ? qg::W8R_RING_BYTES_ONE : qg::W8R_RING_BYTES}, none{0, 0};
  const bool uncut = tokens <= 64 && k_blocks > 10 && tiles <= sms;
  return tokens <= 48 || uncut || 25 * saved(S) > 3 * (tokens - 40) + 50 ? plan : none;
}

// Whether two CTAs per tile of 256 x 256 (PAIR of w8a8.cuh) are faster than one per tile of 128 x 256 or 128 x 128.  Counted in
// rounds of 128 x 256 tiles over the SMs: a last round that is cut in half-width items counts 0.6, a round of 128 x 128 tiles
// 0.5, a round of pairs 0.76; the pairs' longer start and hand-over of a tile count the less the longer K is.  Both ways in turn
// over 370 shapes (1 .. 16 problems of 160 .. 4096 rows, K 512 .. 8192, N 512 .. 14336, both layouts): the choice is 0.1 % behind
// the better one in the mean, 11 % at worst (16 x 279 x 5664 x 13136 468 / 521, seconds at the power limit); constants that were
// fitted to an earlier kernel and K from 2048 on only were 4.4 % and 33 % behind.  us, one / two CTAs per tile: 4096 x 4096 x 14336
// 166 / 148, 2026 x 2464 x 12912 62.6 / 50.6, 14 x 2283 x 1024 x 7568 284 / 227, 12 x 2065 x 672 x 560 22.7 / 20.1, 2228 x 5152 x 3632
// 41.6 / 34.7; not taken: 169 x 800 x 4400 6.6 / 8.0, and, though as fast, 602 x 2048 x 13776 24.0 / 23.2.  QGEMM_W8_PAIR=0 disables it.
static bool w8_pair_pays(int64_t batch, int64_t M, int64_t N, int64_t k_blocks, bool kn, int64_t sms) {
  static const int pair_on = getenv("QGEMM_W8_PAIR") ? atoi(getenv("QGEMM_W8_PAIR")) : 1;
  if (!pair_on || N <= 128) return false;
  auto rounds = [](int64_t tiles, int64_t workers, bool halves) {
    const int64_t whole = tiles / workers, left = tiles % workers;
    return (double)whole + (left == 0 ? 0.0 : (halves && whole != 0 && 2 * left <= workers ? 0.6 : 1.0));
  };
  const int64_t row_blocks = (M + 127) / 128, tiles256 = batch * row_blocks * ((N + 255) / 256);
  const double one = tiles256 >= sms ? rounds(tiles256, sms, kn) : 0.5 * rounds(batch * row_blocks * ((N + 127) / 128), sms, false);
  const double two = rounds(batch * ((M + 255) / 256) * ((N + 255) / 256), sms / 2, true);
  return two * (0.76 + 0.5 / (double)k_blocks) + 1.2 / (double)k_blocks < one;
}

// Plain / batched form: meta == nullptr.  Grouped form: A and C are single [M, K] / [M, N] stacks, B holds
// `batch` (= groups) matrices and `meta` lists num_blocks row blocks (group, first row, valid rows).
static int w8a8_impl(const int8_t* A, const int8_t* B, const float* scale_b, const float* scale_a, void* C,
                     int32_t* acc_out, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t scale_b_len,
                     int64_t scale_a_len, int out_dtype, int b_layout, uint32_t* status, void* stream,
                     const int* meta, int64_t num_blocks, bool zero_uncovered = false) {
  const int64_t batchA = meta ? 1 : batch;  // batch extent of A, C and scale_a
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return fail("qgemm_w8a8: batch, M, N, K must be positive (got %lld, %lld, %lld, %lld)", (long long)batch, (long long)M, (long long)N, (long long)K);
  if (M > (1ll << 30) || N > (1ll << 30) || K > (1ll << 30) || batch > 65535) return fail("qgemm_w8a8: dimension too large");
  if (A == nullptr || B == nullptr) return fail("qgemm_w8a8: A and B must not be null");
  if (b_layout != QGEMM_B_KN && b_layout != QGEMM_B_NK) return fail("qgemm_w8a8: unknown b_layout %d", b_layout);
  if (out_dtype == QGEMM_DT_I32) {
    if (C == nullptr) return fail("qgemm_w8a8: int32 output needs C");
    if (acc_out != nullptr) return fail("qgemm_w8a8: with int32 output pass the buffer as C and acc_out = NULL");
    acc_out = static_cast<int32_t*>(C);
    C = nullptr;
  } else if (out_dtype == QGEMM_DT_F16 || out_dtype == QGEMM_DT_BF16) {
    if (C == nullptr && acc_out == nullptr) return fail("qgemm_w8a8: neither C nor acc_out given");
    if (C != nullptr) {
      if (scale_b == nullptr) return fail("qgemm_w8a8: scale_b must not be null");
      if (scale_b_len != 1 && scale_b_len != N && scale_b_len != batch * N) return fail("qgemm_w8a8: scale_b_len must be 1, N or batch*N (got %lld)", (long long)scale_b_len);
      if (scale_a != nullptr && scale_a_len != M && scale_a_len != batchA * M) return fail("qgemm_w8a8: scale_a_len must be M or batch*M (got %lld)", (long long)scale_a_len);
    }
  } else {
    return fail("qgemm_w8a8: out_dtype must be F16, BF16 or I32 (got %d)", out_dtype);
  }
  if (K % 16 != 0 || N % 16 != 0) return fail("qgemm_w8a8: K and N must be multiples of 16 (got K=%lld, N=%lld)", (long long)K, (long long)N);
  if (!aligned16(A) || !aligned16(B) || !aligned16(C) || !aligned16(acc_out)) return fail("qgemm_w8a8: A, B, C and acc_out must be 16-byte aligned");

  int sms = 0;
  if (ensure_device(&sms)) return -1;

  CUtensorMap tmA, tmB;
  const int64_t k_blocks = (K + 127) / 128, n_tiles128 = (N + 127) / 128, row_tiles = (M + qg::W8R_MAX_MT - 1) / qg::W8R_MAX_MT;
  W8RowsPlan rows_plan{0, 0};
  if (meta == nullptr && acc_out == nullptr)
    rows_plan = w8_rows_plan(batch * n_tiles128 * row_tiles, k_blocks, (M + row_tiles - 1) / row_tiles, b_layout == QGEMM_B_KN, sms);
  const int S = rows_plan.split;
  if (S > 0) {
    const int64_t n_tiles = n_tiles128, m_tiles = row_tiles, tiles = batch * n_tiles * m_tiles;
    if (tiles > 0x7fffffff / qg::W8R_MAX_SPLIT) return fail("qgemm_w8a8: too many tiles");
    const int unit = S == 8 ? 32 : 16;
    qg::W8RowsParams p;
    p.scale_b = scale_b;
    p.scale_a = scale_a;
    p.C = C;
    p.M = (int)M;
    p.N = (int)N;
    p.sb_mode = (scale_b_len == 1) ? 0 : ((scale_b_len == N) ? 1 : 2);
    p.sa_mode = (scale_a == nullptr) ? 0 : ((scale_a_len == M) ? 1 : 2);
    p.n_tiles = (int)n_tiles;
    p.k_blocks = (int)k_blocks;
    p.m_tiles = (int)m_tiles;
    p.mt = (int)(((M + m_tiles - 1) / m_tiles + unit - 1) / unit * unit);
    p.tmem_cols = p.mt <= 32 ? 32 : (p.mt <= 64 ? 64 : 128);
    p.ring = rows_plan.ring;
    p.status = status;
    p.wait_limit_ns = g_wait_limit_ns;
    const uint64_t dims_a[3] = {(uint64_t)K, (uint64_t)M, (uint64_t)batch};
    const uint64_t str_a[2] = {(uint64_t)K, (uint64_t)M * (uint64_t)K};
    const uint32_t box_a[3] = {128, (uint32_t)p.mt, 1};
    if (encode_map(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, A, dims_a, str_a, box_a, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    const bool nk = b_layout == QGEMM_B_NK;
    const uint64_t dims_b[3] = {(uint64_t)(nk ? K : N), (uint64_t)(nk ? N : K), (uint64_t)batch};
    const uint64_t str_b[2] = {(uint64_t)(nk ? K : N), (uint64_t)N * (uint64_t)K};
    const uint32_t box_b[3] = {128, 128, 1};
    if (encode_map(&tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, B, dims_b, str_b, box_b, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    const int grid = (int)(tiles * S);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool bf = out_dtype == QGEMM_DT_BF16;
    if (nk) return bf ? launch_w8_rows<true, true>(tmA, tmB, p, grid, S, s) : launch_w8_rows<true, false>(tmA, tmB, p, grid, S, s);
    return bf ? launch_w8_rows<false, true>(tmA, tmB, p, grid, S, s) : launch_w8_rows<false, false>(tmA, tmB, p, grid, S, s);
  }
  {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)M, (uint64_t)batchA};
    const uint64_t str[2] = {(uint64_t)K, (uint64_t)M * (uint64_t)K};
    const uint32_t box[3] = {128, 128, 1};
    if (encode_map(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, A, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }
  const int64_t row_blocks = meta ? num_blocks : (M + 127) / 128;
  const int64_t tiles256 = batchA * row_blocks * ((N + 255) / 256);
  // A very long K and fewer 128-wide tiles than half the SMs, weights [K, N]: split K over pairs of CTAs (one tile of 256 columns per
  // pair).  Everything else of few tiles is faster by tiles of 128 columns, whose pipeline is six stages deep.  us, split / 128-wide:
  // 256-row problems of 51 tiles, K = 7296 23.0 / 26.8, 63 tiles, K = 8192 22.0 / 24.2, but 24 tiles, K = 5504 21.6 / 22.0; not taken: 40
  // tiles, K = 6656, [N, K] 17.9 / 16.8, 99 tiles, K = 4352 18.3 / 15.1, 114 tiles, K = 4992 18.4 / 15.7.  Without accumulators the
  // few-token form takes these shapes.  QGEMM_W8_SPLITK=0 disables it.
  static const int splitk_on = getenv("QGEMM_W8_SPLITK") ? atoi(getenv("QGEMM_W8_SPLITK")) : 1;
  const bool use_splitk = splitk_on && meta == nullptr && b_layout == QGEMM_B_KN && N > 128 && 2 * batchA * row_blocks * n_tiles128 <= sms && k_blocks >= 50;
  // Otherwise two CTAs per tile of 256 x 256 where that is the faster one (w8_pair_pays).
  const bool use_pair = meta == nullptr && !use_splitk && w8_pair_pays(batch, M, N, k_blocks, b_layout == QGEMM_B_KN, sms);
  const int BN = (N > 128 && (tiles256 >= sms || use_splitk || use_pair)) ? 256 : 128;
  const int64_t m_tiles = use_pair ? (M + 255) / 256 : row_blocks;  // of 128 rows, of 256 for two CTAs
  // Tiles are BN columns wide: narrower ones that fill the last round of the persistent grid better were slower (224 instead of
  // 256 columns on the 4096 x 4096 x 14336 shape, by an earlier form of the kernel: 235 us against 231), and the epilogue wants
  // multiples of 128.
  if (b_layout == QGEMM_B_KN) {
    const uint64_t dims[3] = {(uint64_t)N, (uint64_t)K, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)N, (uint64_t)K * (uint64_t)N};
    const uint32_t box[3] = {128, 128, 1};
    if (encode_map(&tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, B, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  } else {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)N, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)K, (uint64_t)N * (uint64_t)K};
    const uint32_t box[3] = {128, (uint32_t)(use_pair ? 128 : BN), 1};
    if (encode_map(&tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, B, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }

  // C as a tensor map for the epilogue's tiled stores: boxes of 64 outputs x 32 rows, 128-byte swizzle.
  CUtensorMap tmC = tmA;
  static const int tma_store_on = getenv("QGEMM_W8_TMA_STORE") ? atoi(getenv("QGEMM_W8_TMA_STORE")) : 1;  // 0: per-row stores
  const bool tma_store = tma_store_on && C != nullptr;
  if (tma_store) {
    const uint64_t dims[3] = {(uint64_t)N, (uint64_t)M, (uint64_t)batchA};
    const uint64_t str[2] = {(uint64_t)N * 2, (uint64_t)M * (uint64_t)N * 2};
    const uint32_t box[3] = {64, 32, 1};
    if (encode_map(&tmC, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, C, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }

  qg::W8A8Params p;
  p.tma_store = tma_store ? 1 : 0;
  p.scale_b = scale_b;
  p.scale_a = scale_a;
  p.C = C;
  p.acc_out = acc_out;
  p.batch = (int)batchA;
  p.meta = meta;
  p.num_blocks = meta ? (int)num_blocks : 0;
  p.zero_uncovered = zero_uncovered && C != nullptr ? 1 : 0;
  p.groups = (int)batch;
  p.M = (int)M;
  p.N = (int)N;
  p.K = (int)K;
  p.sb_mode = (scale_b_len == 1) ? 0 : ((scale_b_len == N) ? 1 : 2);
  p.sa_mode = (scale_a == nullptr) ? 0 : ((scale_a_len == M) ? 1 : 2);
  p.m_tiles = (int)m_tiles;
  p.group_m = use_pair ? (w8_group_m(2 * m_tiles, K, 0, 0) + 1) / 2 : w8_group_m(m_tiles, K, meta ? batch : 0, N * K);
  p.n_tiles = (int)((N + BN - 1) / BN);
  p.bn = BN;
  const int64_t num_tiles = batchA * p.m_tiles * p.n_tiles;
  if (num_tiles > 0x7fffffff) return fail("qgemm_w8a8: too many tiles");
  p.num_tiles = (int)num_tiles;
  p.k_blocks = (int)((K + 127) / 128);
  p.status = status;
  p.wait_limit_ns = g_wait_limit_ns;
  p.withhold = g_withhold;
  // with rows that no block can cover, a CTA per SM to clear them, whatever the number of tiles
  const bool sure_to_clear = p.zero_uncovered && M > num_blocks * qg::W8_BM;
  const int workers = use_pair ? sms / 2 : sms;  // CTAs, or pairs of them
  const int grid = (int)(num_tiles < workers && !sure_to_clear ? num_tiles : workers);
  // Tail split: when the last round of the persistent grid would run R < grid/2 tiles, those tiles are issued
  // as 2R half-width items instead ([K, N] layout, 256-column tiles).
  p.split_from = p.num_items = p.num_tiles;
  {
    static const int tail_split = getenv("QGEMM_W8_TAIL_SPLIT") ? atoi(getenv("QGEMM_W8_TAIL_SPLIT")) : 1;
    const int64_t R = num_tiles % grid;
    if (tail_split && (use_pair || b_layout == QGEMM_B_KN) && BN == 256 && num_tiles > grid && R > 0 && 2 * R <= grid) {
      p.split_from = (int)(num_tiles - R);
      p.num_items = (int)(num_tiles + R);
    }
  }
  // The next kernel's CTAs then come to the SMs in the order in which these become free.  Grouped calls of several rounds, whose
  // neighbouring CTAs share tiles of L2, lose more by that than a late start costs: 16 groups, 8192 x 7168 x 2048 120.6 us, 126.0 with
  // it, 25 groups, 3751 x 4992 x 3664 118.4 / 120.5, of two rounds 9 groups, 6844 x 2464 x 1232 31.6 / 32.2; of one round 14 groups, 150 x
  // 4256 x 1568 26.2 / 25.5, or of tiles of 128 columns, 17 groups, 1903 x 1184 x 1216 12.2 / 11.5.  Plain and batched calls gain
  // throughout: 1097 x 2496 x 1680 11.7 / 10.9, 519 x 1344 x 2400 7.2 / 6.6, and with the quantiser in front 300 x 2048 x 4096 13.6 / 12.1
  // (calls of 100 us and more by no more than repeats differ).
  p.early = meta == nullptr || BN == 128 || p.num_items <= grid ? 1 : 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool nk = b_layout == QGEMM_B_NK;
  const bool bf = out_dtype == QGEMM_DT_BF16;
  if (use_splitk) {  // [K, N] only
    constexpr auto form = qg::W8_SPLITK;
    return bf ? launch_w8_clusters<false, true, form>(tmA, tmB, tmC, p, (int)num_tiles, s) : launch_w8_clusters<false, false, form>(tmA, tmB, tmC, p, (int)num_tiles, s);
  }
  if (use_pair) {
    constexpr auto form = qg::W8_PAIR;
    if (nk) return bf ? launch_w8_clusters<true, true, form>(tmA, tmB, tmC, p, grid, s) : launch_w8_clusters<true, false, form>(tmA, tmB, tmC, p, grid, s);
    return bf ? launch_w8_clusters<false, true, form>(tmA, tmB, tmC, p, grid, s) : launch_w8_clusters<false, false, form>(tmA, tmB, tmC, p, grid, s);
  }
  if (BN == 256) {
    if (nk) return bf ? launch_w8<256, true, true>(tmA, tmB, tmC, p, grid, s) : launch_w8<256, true, false>(tmA, tmB, tmC, p, grid, s);
    return bf ? launch_w8<256, false, true>(tmA, tmB, tmC, p, grid, s) : launch_w8<256, false, false>(tmA, tmB, tmC, p, grid, s);
  }
  if (nk) return bf ? launch_w8<128, true, true>(tmA, tmB, tmC, p, grid, s) : launch_w8<128, true, false>(tmA, tmB, tmC, p, grid, s);
  return bf ? launch_w8<128, false, true>(tmA, tmB, tmC, p, grid, s) : launch_w8<128, false, false>(tmA, tmB, tmC, p, grid, s);
}

int qgemm_w8a8(const int8_t* A, const int8_t* B, const float* scale_b, const float* scale_a, void* C,
               int32_t* acc_out, int64_t batch, int64_t M, int64_t N, int64_t K, int64_t scale_b_len,
               int64_t scale_a_len, int out_dtype, int b_layout, uint32_t* status, void* stream) {
  return w8a8_impl(A, B, scale_b, scale_a, C, acc_out, batch, M, N, K, scale_b_len, scale_a_len, out_dtype, b_layout,
                   status, stream, nullptr, 0);
}

static int w8a8_grouped_impl(const int8_t* A, const int8_t* B, const float* scale_b, const float* scale_a, void* C,
                             int32_t* acc_out, const int32_t* block_metadata, int64_t num_blocks, int64_t groups,
                             int64_t total_M, int64_t N, int64_t K, int64_t scale_b_len, int64_t scale_a_len, int out_dtype,
                             int b_layout, uint32_t* status, void* stream, bool zero_uncovered) {
  if (num_blocks < 0) return fail("qgemm_w8a8_grouped: num_blocks must not be negative (got %lld)", (long long)num_blocks);
  if (total_M == 0) return 0;  // no rows: nothing to compute
  if (num_blocks == 0) {       // no row is covered
    if (zero_uncovered && C != nullptr && total_M > 0 && N > 0)
      CUDA_OK(cudaMemsetAsync(C, 0, (size_t)total_M * (size_t)N * (out_dtype == QGEMM_DT_I32 ? 4 : 2), static_cast<cudaStream_t>(stream)));
    return 0;
  }
  if (block_metadata == nullptr) return fail("qgemm_w8a8_grouped: block_metadata must not be null");
  if ((reinterpret_cast<uintptr_t>(block_metadata) & 3u) != 0) return fail("qgemm_w8a8_grouped: block_metadata must be 4-byte aligned");
  if (num_blocks > (1ll << 24)) return fail("qgemm_w8a8_grouped: too many row blocks (%lld)", (long long)num_blocks);
  return w8a8_impl(A, B, scale_b, scale_a, C, acc_out, groups, total_M, N, K, scale_b_len, scale_a_len, out_dtype,
                   b_layout, status, stream, block_metadata, num_blocks, zero_uncovered);
}

int qgemm_w8a8_grouped(const int8_t* A, const int8_t* B, const float* scale_b, const float* scale_a, void* C,
                       int32_t* acc_out, const int32_t* block_metadata, int64_t num_blocks, int64_t groups,
                       int64_t total_M, int64_t N, int64_t K, int64_t scale_b_len, int64_t scale_a_len, int out_dtype,
                       int b_layout, uint32_t* status, void* stream) {
  return w8a8_grouped_impl(A, B, scale_b, scale_a, C, acc_out, block_metadata, num_blocks, groups, total_M, N, K, scale_b_len,
                           scale_a_len, out_dtype, b_layout, status, stream, false);
}

int qgemm_w8a8_grouped_zeroed(const int8_t* A, const int8_t* B, const float* scale_b, const float* scale_a, void* C,
                              int32_t* acc_out, const int32_t* block_metadata, int64_t num_blocks, int64_t groups,
                              int64_t total_M, int64_t N, int64_t K, int64_t scale_b_len, int64_t scale_a_len,
                              int out_dtype, int b_layout, uint32_t* status, void* stream) {
  return w8a8_grouped_impl(A, B, scale_b, scale_a, C, acc_out, block_metadata, num_blocks, groups, total_M, N, K, scale_b_len,
                           scale_a_len, out_dtype, b_layout, status, stream, true);
}

int64_t qgemm_w4a16_counter_bytes(void) { return kW4CounterBytes; }

// Wide tiles (w4a16_wide.cuh): the tile's tokens and the cut of the work.  Of the cuts into equal tiles (48 .. 256 tokens,
// a multiple of 16 or, with two CTAs, of 32, fewer when there are fewer tokens) and of three ways to deal T tiles to G CTAs the one with the
// smallest estimated time: whole tiles only; whole rounds of G tiles and each tile of the remainder cut into S equal K
// ranges for S CTAs; or the remainder (with one whole round, when it is small) cut evenly over all CTAs.  The estimate is
// fitted to a sweep of tile heights and cuts over K = 1024 .. 8192, N = 1024 .. 14336, 80 .. 2048 tokens (us): a slab
// 0.95, from about 96 tokens on 0.5 + 0.0048 per token; a tile's end 2 + 0.015 per token; the sum of a tile that S CTAs
// share 2 + S (0.3 + 0.011 per token), or 2 where whole tiles follow behind which it runs; the even cut, where a CTA can
// hold two partial tiles, 3 + 0.06 per token, or 6.  So large problems take the tallest tiles, problems of fewer tiles
// than SMs shorter ones (512 x 2048 x 4096: 128 tiles of 128 tokens 16.4 us, 64 tiles of 256 cut in two 25.5 us), and a
// cut along K is for few tiles of long K (128 x 8192 x 2048: 32 tiles of 64 tokens cut in four 23.3 us, whole 38.6 us).
// Beside whole rounds, and below K = 8192, a remainder is cut in two only: with four or more shares the sums, of tall tiles with
// one accumulator, set the pace (1040 x 1024 x 8192: 41 us, whole tiles 27; 1700 x 4096 x 3072 53 / 43; but 4096 x 8192 x 28672
// in four 1641, in two 1652).
struct W4WidePlan {
  int mt = 0, sk_tiles = 0, sk_grid = 1;
  bool pair = false;
  double time = 0.0;  // estimated
};
static W4WidePlan w4_wide_plan_for(int64_t M, int64_t weight_tiles, int64_t KS, int64_t G, int64_t step) {
  W4WidePlan best;
  if (M <= 0 || weight_tiles <= 0 || KS <= 0) return best;  // a size query about an empty problem
  for (int64_t t = (M + qg::W4W_MAX_MT - 1) / qg::W4W_MAX_MT;; ++t) {
    const int64_t mt = ((M + t - 1) / t + step - 1) / step * step;
    const int64_t tiles = weight_tiles * ((M + mt - 1) / mt), rounds = tiles / G, r = tiles % G;
    const double slab = std::max(0.95, 0.5 + 0.0048 * (double)mt), end = 2.0 + 0.015 * (double)mt;
    auto consider = [&](double slabs, double extra, int64_t sk_tiles, int64_t sk_grid) {
      const double time = slabs * slab + end + extra;
      if (best.mt != 0 && time >= best.time) return;
      best.time = time;
      best.mt = (int)mt;
      best.sk_tiles = (int)sk_tiles;
      best.sk_grid = (int)sk_grid;
    };
    consider((double)((rounds + (r != 0 ? 1 : 0)) * KS), 0.0, 0, 1);
    if (r != 0) {
      for (int64_t S = 2; S <= (rounds != 0 && KS < 32 ? 2 : 8) && S * r <= G && S <= KS; S += 2)
        consider((double)(rounds * KS + (KS + S - 1) / S), rounds != 0 ? 2.0 : 2.0 + (double)S * (0.3 + 0.011 * (double)mt), r, r * S);
      const int64_t sk = r + (rounds != 0 && 2 * r < G ? G : 0);
      if (sk * KS >= G) consider((double)(tiles * KS) / (double)G, rounds != 0 ? 6.0 : 3.0 + 0.06 * (double)mt, sk, G);
    }
    if (mt <= 48 || tiles > 4 * G) break;  // more tiles than that only convert the weights more often
  }
  return best;
}
// On G SMs: by single CTAs, or by pairs of them with tiles of 256 weight rows.  A pair halves what a CTA loads of the activations,
// which counts from tiles of about 192 tokens on; each hand-over between the two CTAs takes longer, once per launch and once per
// tile, and a tile of few slabs does not earn that back: 0.93 of the time, 2.5 us and 0.4 us per tile of a pair, from 13 slabs on.
// Fitted to and checked on 265 shapes, K 1024 .. 8192, N 1024 .. 28672, 180 .. 4096 tokens, both ways in turn: 88 take pairs, four
// of them 0.8 .. 1.6 % slower than one CTA, the mean 3.5 % faster.  us, one CTA / two: 4096 x 8192 x 28672 1448 / 1389, 500 x 8192
// x 28672 184 / 174, 2235 x 4096 x 17440 260 / 247; not taken: 2286 x 2816 x 16576 175 / 171, 3314 x 2560 x 8736 130 / 134, 2628 x
// 2048 x 21520 205 / 208, 1152 x 1536 x 13792 55.3 / 60.2, 3468 x 1024 x 25408 194 / 204.  QGEMM_W4_PAIR=0 disables pairs.
static W4WidePlan w4_wide_plan(int64_t M, int64_t batch, int64_t N, int64_t KS, int64_t G, bool pairs = true) {
  static const int pair_on = getenv("QGEMM_W4_PAIR") ? atoi(getenv("QGEMM_W4_PAIR")) : 1;
  const W4WidePlan one = w4_wide_plan_for(M, batch * ((N + 127) / 128), KS, G, qg::W4W_MT_STEP);
  if (!pairs || !pair_on || G < 2 || one.mt == 0 || KS < 13) return one;
  const int64_t weight_tiles = batch * ((N + 255) / 256);
  W4WidePlan two = w4_wide_plan_for(M, weight_tiles, KS, G / 2, qg::W4W_PAIR_MT_STEP);
  two.pair = true;
  const double tiles_each = (double)(weight_tiles * ((M + two.mt - 1) / two.mt)) / (double)(G / 2);
  return two.mt >= 192 && 0.93 * two.time + 2.5 + 0.4 * tiles_each < one.time ? two : one;
}
// Scratch for tiles of mt tokens: arrival counters, two partial sums per CTA, the prepared activations.
static int64_t w4_wide_bytes(int64_t batch, int64_t M, int64_t K, int64_t grid, int mt) {
  return kW4CounterBytes + grid * 2 * (int64_t)mt * 128 * 4 + batch * M * K * 2;
}
static int64_t w4_wide_workspace_bytes(int64_t batch, int64_t M, int64_t N, int64_t K) {
  int sms = 0;
  if (ensure_device(&sms)) return -1;
  const int64_t grid = sms < kW4MaxGrid ? sms : kW4MaxGrid;
  return w4_wide_bytes(batch, M, K, grid, w4_wide_plan(M, batch, N, (K + 255) / 256, grid).mt);
}

// Which of the W4A16 kernels takes a call: the group-sum kernel (w4a16_gs.cuh) up to 64 tokens where it can (wide scale
// groups, scalar zero point or a zeros tensor of mode "quantized"); scale groups of 32 / 64 up to 16 tokens the
// register-operand decode kernel (up to 8) and w4a16.cuh; everything else the wide tiles.  Groups of 64, K = 8192, N =
// 28672: at 16 tokens 46.9 us (w4a16.cuh) against 54.2 (wide), at 24 56.6 against 53.7; K = N = 4096 at 24: 16.1
// against 12.1, at 64: 23.9 against 15.6.
enum W4Route { W4_GROUP_SUM, W4_NARROW_GROUPS, W4_WIDE };
static W4Route w4_route(int64_t M, int64_t K, int64_t group, bool has_scales, bool zeros_tensor, int zero_mode) {
  const bool gs = w4_gs_shape_ok(M, has_scales, group, K);
  if (zeros_tensor) return gs && zero_mode == QGEMM_ZERO_QUANTIZED ? W4_GROUP_SUM : W4_WIDE;
  if (gs) return W4_GROUP_SUM;
  return M <= 16 ? W4_NARROW_GROUPS : W4_WIDE;
}

// Scratch of the kernels for few tokens: the arrival counters first (fixed place whatever the tile height), then two
// partial slots of [MT][128] fp32 per CTA, then the prepared activations - plain f16 [M, K] in the kernel's K order, or
// in blocks of 64 k for the group-sum kernel (counted with its token tile).
static int64_t w4_workspace_bytes(int64_t batch, int64_t M, int64_t N, int64_t K) {
  int sms = 0;
  if (ensure_device(&sms)) return -1;
  const int64_t grid = sms < kW4MaxGrid ? sms : kW4MaxGrid;
  // sized for whichever small-token kernel the scale groups will select (the group-sum kernel's tile is the taller)
  const int mt = M <= 64 ? w4_pick_mt(M, true) : 128;
  int64_t a_bytes = batch * M * K * 2;
  if (M <= 64) {
    const int64_t images = batch * ((K + 255) / 256) * 2 * (int64_t)qg::w4g_half_bytes(mt);
    if (images > a_bytes) a_bytes = images;
  }
  return kW4CounterBytes + grid * 2 * (int64_t)mt * 128 * 4 + a_bytes;
}

int64_t qgemm_w4a16_batched_workspace_bytes(int64_t batch, int64_t M, int64_t N, int64_t K) {
  const int64_t few = w4_workspace_bytes(batch, M, N, K);
  return few < 0 ? -1 : std::max(few, w4_wide_workspace_bytes(batch, M, N, K));
}

int64_t qgemm_w4a16_ex_workspace_bytes(int64_t batch, int64_t M, int64_t N, int64_t K, int has_zeros_tensor) {
  (void)has_zeros_tensor;  // zero points are taken in flight
  return qgemm_w4a16_batched_workspace_bytes(batch, M, N, K);
}

int64_t qgemm_w4a16_call_workspace_bytes(int64_t batch, int64_t M, int64_t N, int64_t K, int64_t group, int has_scales,
                                         int has_zeros_tensor, int zero_mode) {
  if (w4_route(M, K, group, has_scales != 0, has_scales && has_zeros_tensor, zero_mode) == W4_WIDE)
    return w4_wide_workspace_bytes(batch, M, N, K);
  return w4_workspace_bytes(batch, M, N, K);
}

int64_t qgemm_w4a16_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  return qgemm_w4a16_batched_workspace_bytes(1, M, N, K);
}

// Destinations of the gathered form: `n` row-major [M, ldc] buffers (one per rank, peers' buffers mapped into this
// process), this rank's columns starting at col0.
struct GatherDst {
  void* const* dst;
  int n;
  int64_t ldc, col0;
};

int qgemm_w4a16(const void* A, const uint8_t* B_packed, const void* scales, int zero, int64_t group, void* C,
                void* workspace, int64_t workspace_bytes, int64_t M, int64_t N, int64_t K, int a_dtype,
                int out_dtype, uint32_t* status, void* stream) {
  return qgemm_w4a16_batched(A, B_packed, scales, zero, group, C, workspace, workspace_bytes, 1, M, N, K, a_dtype,
                             out_dtype, status, stream);
}

static int w4a16_impl(const void* A, const uint8_t* B_packed, const void* scales, int zero, int64_t group, void* C,
                      void* workspace, int64_t workspace_bytes, int64_t batch, int64_t M, int64_t N, int64_t K,
                      int a_dtype, int out_dtype, uint32_t* status, void* stream, const void* zeros, int zero_mode,
                      int weight_format, const GatherDst* gd = nullptr);

int qgemm_w4a16_batched(const void* A, const uint8_t* B_packed, const void* scales, int zero, int64_t group, void* C,
                        void* workspace, int64_t workspace_bytes, int64_t batch, int64_t M, int64_t N, int64_t K,
                        int a_dtype, int out_dtype, uint32_t* status, void* stream) {
  return w4a16_impl(A, B_packed, scales, zero, group, C, workspace, workspace_bytes, batch, M, N, K, a_dtype, out_dtype,
                    status, stream, nullptr, QGEMM_ZERO_ORIGINAL, QGEMM_W4_SEQUENTIAL);
}

int qgemm_w4a16_ex(const void* A, const uint8_t* B_packed, const void* scales, const void* zeros, int zero,
                   int zero_mode, int weight_format, int64_t group, void* C, void* workspace, int64_t workspace_bytes,
                   int64_t batch, int64_t M, int64_t N, int64_t K, int a_dtype, int out_dtype, uint32_t* status,
                   void* stream) {
  if (weight_format != QGEMM_W4_SEQUENTIAL && weight_format != QGEMM_W4_INTERLEAVED_F16)
    return fail("qgemm_w4a16_ex: unknown weight_format %d", weight_format);
  if (zero_mode != QGEMM_ZERO_ORIGINAL && zero_mode != QGEMM_ZERO_RESCALE && zero_mode != QGEMM_ZERO_QUANTIZED)
    return fail("qgemm_w4a16_ex: unknown zero_mode %d", zero_mode);
  if (zeros == nullptr && zero_mode == QGEMM_ZERO_RESCALE)
    return fail("qgemm_w4a16_ex: zero mode 'rescale' needs the zeros tensor");
  if (zeros != nullptr) {
    if (scales == nullptr) return fail("qgemm_w4a16_ex: a zeros tensor needs scales");
    if (!aligned16(zeros)) return fail("qgemm_w4a16_ex: zeros must be 16-byte aligned");
    if (N % 16 != 0) return fail("qgemm_w4a16_ex: a zeros tensor needs N to be a multiple of 16 (got %lld)", (long long)N);
  }
  return w4a16_impl(A, B_packed, scales, zero, group, C, workspace, workspace_bytes, batch, M, N, K, a_dtype, out_dtype,
                    status, stream, zeros, zero_mode, weight_format);
}

static int w4a16_impl(const void* A, const uint8_t* B_packed, const void* scales, int zero, int64_t group, void* C,
                      void* workspace, int64_t workspace_bytes, int64_t batch, int64_t M, int64_t N, int64_t K,
                      int a_dtype, int out_dtype, uint32_t* status, void* stream, const void* zeros, int zero_mode,
                      int weight_format, const GatherDst* gd) {
  if (batch <= 0 || batch > 65535) return fail("qgemm_w4a16: batch must be in 1..65535 (got %lld)", (long long)batch);
  if (M <= 0 || N <= 0 || K <= 0) return fail("qgemm_w4a16: M, N, K must be positive (got %lld, %lld, %lld)", (long long)M, (long long)N, (long long)K);
  if (M > (1ll << 30) || N > (1ll << 30) || K > (1ll << 30)) return fail("qgemm_w4a16: dimension too large");
  if (A == nullptr || B_packed == nullptr || (C == nullptr && gd == nullptr)) return fail("qgemm_w4a16: A, B_packed and C must not be null");
  if (a_dtype != QGEMM_DT_F16 && a_dtype != QGEMM_DT_BF16) return fail("qgemm_w4a16: a_dtype must be F16 or BF16 (got %d)", a_dtype);
  if (out_dtype != QGEMM_DT_F16 && out_dtype != QGEMM_DT_BF16) return fail("qgemm_w4a16: out_dtype must be F16 or BF16 (got %d)", out_dtype);
  if (K % 32 != 0) return fail("qgemm_w4a16: K must be a multiple of 32 (got %lld)", (long long)K);
  if (N % 8 != 0) return fail("qgemm_w4a16: N must be a multiple of 8 (got %lld)", (long long)N);
  if (!aligned16(A) || !aligned16(B_packed) || !aligned16(C) || !aligned16(scales) || !aligned16(workspace)) return fail("qgemm_w4a16: pointers must be 16-byte aligned");
  if (scales != nullptr) {
    if (zero < 0 || zero > 15) return fail("qgemm_w4a16: zero must be in 0..15 (got %d)", zero);
    if (group <= 0 || K % group != 0) return fail("qgemm_w4a16: group must divide K (got group=%lld, K=%lld)", (long long)group, (long long)K);
    const bool ok = (group < 256 && 256 % group == 0 && group >= 32) || (group % 256 == 0) || (group >= K);
    if (!ok) return fail("qgemm_w4a16: group must be 32, 64, 128, a multiple of 256, or the whole K (got %lld)", (long long)group);
  } else {
    zero = 0;
    group = K;
  }
  const W4Route route = w4_route(M, K, group, scales != nullptr, zeros != nullptr, zero_mode);
  const bool use_gs = route == W4_GROUP_SUM, wide = route == W4_WIDE;
  int64_t need = w4_workspace_bytes(batch, M, N, K);
  if (need < 0) return -1;
  int sms = 0;
  if (ensure_device(&sms)) return -1;
  const int64_t grid_max = sms < kW4MaxGrid ? sms : kW4MaxGrid;
  W4WidePlan plan;
  if (wide) {
    plan = w4_wide_plan(M, batch, N, (K + 255) / 256, grid_max);
    // pairs may want taller tiles, and so more scratch: a workspace that does for single CTAs stays good for those
    if (plan.pair && workspace_bytes < w4_wide_bytes(batch, M, K, grid_max, plan.mt)) plan = w4_wide_plan(M, batch, N, (K + 255) / 256, grid_max, false);
  }
  const int64_t wide_need = wide ? w4_wide_bytes(batch, M, K, grid_max, plan.mt) : 0;
  // a workspace too small for the wide tiles' partial sums will do if it has room for 128 tokens': no tile is split then
  if (wide) need = std::min(need, wide_need);
  const bool wide_unsplit = wide && workspace_bytes < wide_need;
  if (workspace == nullptr || workspace_bytes < need) return fail("qgemm_w4a16: workspace of %lld bytes needed (got %lld)", (long long)need, (long long)workspace_bytes);

  if (wide && (plan.mt <= 0 || plan.mt > qg::W4W_MAX_MT || plan.mt % (plan.pair ? qg::W4W_PAIR_MT_STEP : qg::W4W_MT_STEP) != 0)) return fail("qgemm_w4a16: no MMA has %d tokens", plan.mt);
  int mt = wide ? plan.mt : w4_pick_mt(M, use_gs);
  if (gd != nullptr && mt < 16) mt = 16;  // the register-operand decode kernel writes one destination only

  CUtensorMap tmW, tmS, tmZ, tmA;
  memset(&tmS, 0, sizeof(tmS));
  memset(&tmZ, 0, sizeof(tmZ));
  {
    const uint64_t dims[3] = {(uint64_t)(K / 2), (uint64_t)N, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)(K / 2), (uint64_t)N * (uint64_t)(K / 2)};
    const uint32_t box[3] = {128, 128, 1};
    if (encode_map(&tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, B_packed, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }
  // One group for a K below a slab: to the other kernels that is one scale row for the whole slab, whatever K is (256 / K rows
  // are fewer than the K / 32 that a slab's chunks would be dealt to, and those beyond are never fetched).
  const int64_t row_k = !use_gs && group >= K && group < 256 ? 256 : group;
  // the group-sum kernel fetches the scale rows of a slab's two 128-k halves: two rows for groups of 128, else one
  int scale_rows = 1;
  if (scales != nullptr) {
    scale_rows = use_gs ? (group == 128 ? 2 : 1) : (row_k < 256 ? (int)(256 / row_k) : 1);
    const uint64_t dims[3] = {(uint64_t)N, (uint64_t)(K / group), (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)N * 2, (uint64_t)(K / group) * (uint64_t)N * 2};
    const uint32_t box[3] = {128, (uint32_t)scale_rows, 1};
    if (encode_map(&tmS, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, scales, dims, str, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return -1;
    if (zeros != nullptr &&
        encode_map(&tmZ, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, zeros, dims, str, box, CU_TENSOR_MAP_SWIZZLE_NONE))
      return -1;
  }
  uint8_t* a_prepared = static_cast<uint8_t*>(workspace) + kW4CounterBytes + (wide_unsplit ? 0 : grid_max * 2 * (int64_t)mt * 128 * 4);
  if (!use_gs) {
    const uint64_t dims[3] = {(uint64_t)K, (uint64_t)M, (uint64_t)batch};
    const uint64_t str[2] = {(uint64_t)K * 2, (uint64_t)M * (uint64_t)K * 2};
    const uint32_t box[3] = {64, (uint32_t)(plan.pair ? mt / 2 : mt), 1};
    if (encode_map(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, a_prepared, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
  }

  qg::W4A16Params p;
  p.C = C;
  p.n_dst = 0;
  p.ldc = p.col0 = 0;
  for (int d = 0; d < 8; ++d) p.c_dst[d] = nullptr;
  if (gd != nullptr) {
    p.n_dst = gd->n;
    p.ldc = (int)gd->ldc;
    p.col0 = (int)gd->col0;
    for (int d = 0; d < gd->n; ++d) p.c_dst[d] = gd->dst[d];
  }
  p.ws_counters = static_cast<uint32_t*>(workspace);
  p.ws_partials = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + kW4CounterBytes);
  p.M = (int)M;
  p.N = (int)N;
  p.K = (int)K;
  p.group = (int)(row_k > (1 << 30) ? (1 << 30) : row_k);
  p.zero = zero;
  p.has_scales = scales != nullptr;
  p.m_tiles = (int)((M + mt - 1) / mt);
  const int tile_rows = plan.pair ? 256 : 128;  // weight rows
  p.n_tiles = (int)((N + tile_rows - 1) / tile_rows);
  p.batch = (int)batch;
  const int64_t num_tiles = batch * (int64_t)p.m_tiles * p.n_tiles;
  if (num_tiles > 0x3fffffff) return fail("qgemm_w4a16: too many tiles");
  p.num_tiles = (int)num_tiles;
  p.KS = (int)((K + 255) / 256);
  p.scale_rows = scale_rows;
  p.total_items = num_tiles * p.KS;
  p.status = status;
  p.wait_limit_ns = g_wait_limit_ns;
  p.withhold = g_withhold;
  p.A_raw = nullptr;
  p.a_is_bf16 = a_dtype == QGEMM_DT_BF16 ? 1 : 0;
  p.w_interleaved = weight_format == QGEMM_W4_SEQUENTIAL ? 0 : 1;
  int64_t grid = sms < kW4MaxGrid ? sms : kW4MaxGrid;
  if (plan.pair) grid /= 2;  // pairs of CTAs
  if (p.total_items < grid) grid = p.total_items;
  // Small problems (a few slabs per CTA): prefer a smaller grid that cuts every tile into equal K ranges, one per CTA, over an even
  // deal that leaves most CTAs with two partial tiles and so two split-K hand-overs, each of which takes longer than several slabs.
  // The group-sum kernel: down to two fifths of the SMs, as long as a CTA gets no more than five slabs more by it, nine where the
  // tiles are whole and nothing is handed over.  us, even / equal: 16 x 4608 x 1312 12.3 / 8.3 (99 CTAs), 32 x 3072 x 2256 14.2 / 9.4 (108),
  // 20 x 5376 x 1200 16.0 / 10.7 (70), 64 x 6912 x 3040 18.4 / 16.2 (72), whole tiles 64 x 1280 x 7728 14.1 / 8.0 (61), 2 x 20 x 3840 x 3888
  // 12.2 / 11.1 (62); not taken: 8 x 7168 x 5296 11.2 / 11.8 (84 CTAs of 14 slabs instead of 8), 4 x 20 x 6656 x 1088 13.1 / 14.6 (72 of 13).
  // (120 shapes of 1 .. 64 tokens, thirty for each step from three quarters down: 28 % faster in the mean in each.)
  if (!wide && p.total_items <= 8 * grid && p.total_items > grid) {
    const int64_t least = use_gs ? (2 * grid + 4) / 5 : (3 * grid + 3) / 4;
    for (int64_t g2 = grid; g2 >= least; --g2) {
      if (p.total_items % g2 != 0) continue;
      const int64_t per = p.total_items / g2;
      if (p.KS % per == 0 && per * grid - p.total_items <= (per == p.KS ? 9 : 5) * grid) {
        grid = g2;
        break;
      }
    }
  }
  // Group-sum kernel: whole tiles per CTA where there are enough, and only the remainder (plus one round when the
  // remainder alone would give every CTA a sliver of a tile) cut stream-K fashion, processed first, so that its hand-overs
  // run beside the whole tiles' work and the launch ends with plain tile writes.  QGEMM_W4_HYBRID=0 cuts all tiles
  // stream-K fashion.
  p.sk_tiles = p.num_tiles;
  p.sk_grid = 1;
  p.dp_rounds = 0;
  if (wide) {
    p.sk_tiles = wide_unsplit ? 0 : plan.sk_tiles;
    p.sk_grid = plan.sk_grid;
  } else {
    static const int hybrid = getenv("QGEMM_W4_HYBRID") ? atoi(getenv("QGEMM_W4_HYBRID")) : 1;
    const int64_t rounds = num_tiles / grid, r = num_tiles % grid;
    if (hybrid && use_gs && rounds >= 1) {
      const bool borrow = r != 0 && 2 * r < grid;
      p.dp_rounds = (int)(borrow ? rounds - 1 : rounds);
      p.sk_tiles = (int)(borrow ? r + grid : r);
    }
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool bf = out_dtype == QGEMM_DT_BF16;
  // Problems of a few slabs per CTA (16 tokens at most, K <= 4096: every tile's K cut over a cluster of 1, 2 or 4 CTAs
  // with at most four slabs each, all clusters resident at once): one launch, no pre-pass, no scratch - see the
  // kernel's SMALL parameter.  Measured against the two-launch form: 16 x 4096 x 4096 9.2 / 10.6 us, 16 x 2048 x 8192
  // 8.8 / 9.8 us; with more clusters than SMs (several waves) it loses.  QGEMM_W4_SMALL=0 keeps the two-launch form.
  {
    static const int small_on = getenv("QGEMM_W4_SMALL") ? atoi(getenv("QGEMM_W4_SMALL")) : 1;
    if (small_on && use_gs && mt == 16 && gd == nullptr && zeros == nullptr && g_withhold != 1) {
      int cluster = 0;
      for (int c = 1; c <= 4; c *= 2)  // clusters of eight were measured slower than the two-launch form (15.3 / 11.3 us)
        if (p.KS % c == 0 && p.KS / c <= qg::W4G_SMALL_MAX_SLABS) { cluster = c; break; }
      static const int small_waves = getenv("QGEMM_W4_SMALL_WAVES") ? atoi(getenv("QGEMM_W4_SMALL_WAVES")) : 1;
      if (cluster > 0 && num_tiles * cluster <= (int64_t)small_waves * sms) {
        p.A_raw = A;
        return launch_w4g_small(bf, tmW, tmS, p, (int)(num_tiles * cluster), cluster, s);
      }
    }
  }
  if (use_gs) {
    const CUtensorMap* tz = zeros != nullptr ? &tmZ : nullptr;
    const bool a_bf = a_dtype == QGEMM_DT_BF16;
    // prepared activations: [batch][64-k block][M][64], K padded to whole slabs
    const uint64_t dims[3] = {64, (uint64_t)M, (uint64_t)batch * (uint64_t)p.KS * 4};
    const uint64_t str[2] = {128, (uint64_t)M * 128};
    const uint32_t box[3] = {64, (uint32_t)mt, 4};
    if (encode_map(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, a_prepared, dims, str, box, CU_TENSOR_MAP_SWIZZLE_128B)) return -1;
    if (launch_w4g_prepare(A, a_prepared, p, a_bf, sms, s)) return -1;
    if (mt == 16) return launch_w4g<16>(bf, tmW, tmS, tz, tmA, p, (int)grid, s);
    if (mt == 32) return launch_w4g<32>(bf, tmW, tmS, tz, tmA, p, (int)grid, s);
    return launch_w4g<64>(bf, tmW, tmS, tz, tmA, p, (int)grid, s);
  }
  {
    const long long n_chunks = (long long)batch * M * K / 8;
    const long long blocks = (n_chunks + 255) / 256;
    if (blocks > 0x7fffffffll) return fail("qgemm_w4a16: activation tensor too large");
    // Launched as a programmatic dependent too: behind another call of this operator (whose GEMM kernel lets its
    // dependents go at once) the pre-pass is already resident, waiting, when that call ends, and the GEMM kernel
    // behind it sets up and streams its first weights meanwhile.  Behind any other kernel this is plain stream order.
    const uint4* a_in = static_cast<const uint4*>(A);
    uint4* a_out = reinterpret_cast<uint4*>(a_prepared);
    const int is_bf = a_dtype == QGEMM_DT_BF16 ? 1 : 0, permute = weight_format == QGEMM_W4_SEQUENTIAL ? 1 : 0;
    if (launch_pdl(qg::w4a16_prepare_activations, (int)blocks, 256, 0, s, a_in, a_out, n_chunks, is_bf, permute,
                   p.ws_counters, (int)(kW4CounterBytes / 4)))
      return -1;
  }
  if (wide) {
    const CUtensorMap& tz = zeros != nullptr ? tmZ : tmS;
    if (plan.pair) return launch_w4w<true>(bf, zeros != nullptr, tmW, tmS, tz, tmA, p, mt, zero_mode, (int)grid, s);
    return launch_w4w<false>(bf, zeros != nullptr, tmW, tmS, tz, tmA, p, mt, zero_mode, (int)grid, s);
  }
  if (gd == nullptr && w4_use_decode(M) && mt <= 16 && M <= w4_decode_max_m()) {
    if (scales == nullptr) return launch_w4d<0>(bf, mt, tmW, tmS, tmA, p, (int)grid, s);
    if (group >= 128) return launch_w4d<4>(bf, mt, tmW, tmS, tmA, p, (int)grid, s);
    if (group == 64) return launch_w4d<2>(bf, mt, tmW, tmS, tmA, p, (int)grid, s);
    return launch_w4d<1>(bf, mt, tmW, tmS, tmA, p, (int)grid, s);
  }
  return launch_w4(bf, tmW, tmS, tmA, p, (int)grid, s);
}

int qgemm_w4a16_gather(const void* A, const uint8_t* B_packed, const void* scales, int zero, int64_t group,
                       void* const* C_dst, int n_dst, int64_t ldc, int64_t col0, void* workspace,
                       int64_t workspace_bytes, int64_t M, int64_t N, int64_t K, int a_dtype, int out_dtype,
                       uint32_t* status, void* stream) {
  if (C_dst == nullptr || n_dst < 1 || n_dst > 8) return fail("qgemm_w4a16_gather: 1 to 8 destinations required (got %d)", n_dst);
  for (int d = 0; d < n_dst; ++d)
    if (C_dst[d] == nullptr || !aligned16(C_dst[d])) return fail("qgemm_w4a16_gather: destination %d is null or not 16-byte aligned", d);
  if (ldc <= 0 || ldc > (1ll << 30) || col0 < 0 || N <= 0 || col0 + N > ldc)
    return fail("qgemm_w4a16_gather: columns [%lld, %lld) do not fit in rows of %lld", (long long)col0, (long long)(col0 + N), (long long)ldc);
  if (ldc % 8 != 0 || col0 % 8 != 0) return fail("qgemm_w4a16_gather: ldc and col0 must be multiples of 8 (got %lld, %lld)", (long long)ldc, (long long)col0);
  GatherDst gd{C_dst, n_dst, ldc, col0};
  return w4a16_impl(A, B_packed, scales, zero, group, nullptr, workspace, workspace_bytes, 1, M, N, K, a_dtype, out_dtype,
                    status, stream, nullptr, QGEMM_ZERO_ORIGINAL, QGEMM_W4_SEQUENTIAL, &gd);
}

}  // extern "C"

// ---- "my blocks have landed" between the ranks of the gathered form ----
namespace {
struct PeerSlots {
  uint32_t* slot[8];
};
// Thread r: release-store the epoch into this rank's slot of rank r's flag array, then acquire-poll slot r of this
// rank's own array until rank r's epoch has arrived.  Bounded: gives up after limit_ns and reports it.
__global__ void peer_signal_wait_kernel(PeerSlots dst, const uint32_t* local_flags, int n, uint32_t epoch,
                                        uint32_t* epoch_counter, unsigned long long limit_ns, uint32_t* status) {
  __shared__ uint32_t epoch_s;
  const int r = threadIdx.x;
  if (epoch_counter != nullptr) {  // the epoch lives on the device: replays of a captured launch keep counting
    if (r == 0) {
      epoch_s = *epoch_counter + 1u;
      *epoch_counter = epoch_s;
    }
    __syncthreads();
    epoch = epoch_s;
  }
  if (r >= n) return;
  __threadfence_system();
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(dst.slot[r]), "r"(epoch) : "memory");
  const uint32_t* mine = local_flags + r;
  const unsigned long long t0 = qg::global_timer_ns();
  for (;;) {
    uint32_t v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(mine) : "memory");
    if ((int32_t)(v - epoch) >= 0) break;
    if (qg::global_timer_ns() - t0 > limit_ns) {
      if (status != nullptr) atomicMax(status, (uint32_t)qg::ST_TIMEOUT_PEER);
      break;
    }
    __nanosleep(100);
  }
}
}  // namespace

extern "C" {

int qgemm_peer_signal_wait(void* const* flag_slots, int n, const uint32_t* local_flags, uint32_t epoch,
                           uint32_t* epoch_counter, uint32_t* status, void* stream) {
  if (flag_slots == nullptr || local_flags == nullptr || n < 1 || n > 8) return fail("qgemm_peer_signal_wait: 1 to 8 ranks, non-null flag arrays required (got n=%d)", n);
  PeerSlots dst;
  for (int r = 0; r < 8; ++r) dst.slot[r] = nullptr;
  for (int r = 0; r < n; ++r) {
    if (flag_slots[r] == nullptr || (reinterpret_cast<uintptr_t>(flag_slots[r]) & 3u) != 0) return fail("qgemm_peer_signal_wait: flag slot %d is null or misaligned", r);
    dst.slot[r] = static_cast<uint32_t*>(flag_slots[r]);
  }
  peer_signal_wait_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(dst, local_flags, n, epoch, epoch_counter, g_wait_limit_ns, status);
  CUDA_OK(cudaGetLastError());
  return 0;
}

// ---- mapping another process's buffer into this one (same node), for the gathered form ----
static_assert(sizeof(cudaIpcMemHandle_t) == QGEMM_IPC_HANDLE_BYTES, "IPC handle size");

int qgemm_ipc_export(const void* dev_ptr, void* handle_out, int64_t* offset_out) {
  if (dev_ptr == nullptr || handle_out == nullptr || offset_out == nullptr) return fail("qgemm_ipc_export: null argument");
  int sms = 0;
  if (ensure_device(&sms)) return -1;
  // the handle names the whole allocation the pointer lies in; the pointer's offset inside it travels with it
  using RangeFn = CUresult (*)(CUdeviceptr*, size_t*, CUdeviceptr);
  static RangeFn range_fn = nullptr;
  if (range_fn == nullptr) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    CUDA_OK(cudaGetDriverEntryPoint("cuMemGetAddressRange", &fn, cudaEnableDefault, &qres));
    if (qres != cudaDriverEntryPointSuccess || fn == nullptr) return fail("cuMemGetAddressRange not available from the driver");
    range_fn = reinterpret_cast<RangeFn>(fn);
  }
  CUdeviceptr base = 0;
  size_t size = 0;
  const CUresult r = range_fn(&base, &size, reinterpret_cast<CUdeviceptr>(dev_ptr));
  if (r != CUDA_SUCCESS) return fail("cuMemGetAddressRange failed with CUresult %d", (int)r);
  cudaIpcMemHandle_t h;
  CUDA_OK(cudaIpcGetMemHandle(&h, reinterpret_cast<void*>(base)));
  memcpy(handle_out, &h, sizeof(h));
  *offset_out = (int64_t)(reinterpret_cast<CUdeviceptr>(dev_ptr) - base);
  return 0;
}

int qgemm_ipc_open(const void* handle, void** base_out) {
  if (handle == nullptr || base_out == nullptr) return fail("qgemm_ipc_open: null argument");
  cudaIpcMemHandle_t h;
  memcpy(&h, handle, sizeof(h));
  void* ptr = nullptr;
  CUDA_OK(cudaIpcOpenMemHandle(&ptr, h, cudaIpcMemLazyEnablePeerAccess));
  *base_out = ptr;
  return 0;
}

int qgemm_ipc_close(void* base) {
  if (base == nullptr) return 0;
  CUDA_OK(cudaIpcCloseMemHandle(base));
  return 0;
}

int qgemm_unpack_int4(const uint8_t* B_packed, int8_t* out, int64_t N, int64_t K, int signed_nibbles,
                      void* stream) {
  if (N <= 0 || K <= 0 || (K % 2) != 0) return fail("qgemm_unpack_int4: N, K must be positive and K even (got %lld, %lld)", (long long)N, (long long)K);
  if (B_packed == nullptr || out == nullptr) return fail("qgemm_unpack_int4: null pointer");
  if (!aligned16(B_packed) || !aligned16(out)) return fail("qgemm_unpack_int4: pointers must be 16-byte aligned");
  const long long n_bytes = (long long)N * (K / 2);
  const long long threads = (n_bytes + 15) / 16;
  const int block = 256;
  const long long grid = (threads + block - 1) / block;
  if (grid > 0x7fffffffll) return fail("qgemm_unpack_int4: tensor too large");
  unpack_int4_kernel<<<(unsigned)grid, block, 0, static_cast<cudaStream_t>(stream)>>>(B_packed, out, n_bytes, signed_nibbles);
  CUDA_OK(cudaGetLastError());
  return 0;
}

int qgemm_act_quant(const void* X, int8_t* Y, float* S, int64_t M, int64_t N, int x_dtype, int round_scale,
                    void* stream) {
  if (M < 0 || N <= 0 || (N % 8) != 0) return fail("qgemm_act_quant: M >= 0 and N a positive multiple of 8 required (got M=%lld, N=%lld)", (long long)M, (long long)N);
  if (N > (1ll << 30)) return fail("qgemm_act_quant: N too large (%lld)", (long long)N);
  if (x_dtype != QGEMM_DT_F16 && x_dtype != QGEMM_DT_BF16) return fail("qgemm_act_quant: x_dtype must be F16 or BF16 (got %d)", x_dtype);
  if (M == 0) return 0;
  if (X == nullptr || Y == nullptr || S == nullptr) return fail("qgemm_act_quant: null pointer");
  if (!aligned16(X) || (reinterpret_cast<uintptr_t>(Y) & 7u) != 0 || (reinterpret_cast<uintptr_t>(S) & 3u) != 0)
    return fail("qgemm_act_quant: X must be 16-byte, Y 8-byte and S 4-byte aligned");
  qg::ActQuantParams p;
  p.X = static_cast<const uint4*>(X);
  p.Y = Y;
  p.S = S;
  p.M = M;
  p.N = (int)N;
  p.is_bf16 = x_dtype == QGEMM_DT_BF16;
  p.round_scale = round_scale != 0;
  const int64_t chunks = N / 8;
  int sms = 0;
  if (ensure_device(&sms)) return -1;
  // Threads per row.  While the rows leave threads idle, latency counts, and what a thread does one after another: one chunk each in
  // rows of up to 512 chunks, else two, as long as that is no more than about half of the threads that the SMs hold.  Above that the
  // fewest of 32..256 that keep a row in at most 4 chunks per thread (8 at 256).  us, four / two / one chunk per thread: 24 x 4096
  // 2.74 / 1.95 / 1.78, 148 x 1024 2.70 / 1.98 / 1.72, 600 x 2048 3.66 / 2.85 / 2.73, 1200 x 2048 4.81 / 3.60 / 3.97, 300 x 8192 4.25 / 3.81 /
  // 6.05, 148 x 14336 4.66 / 3.43 / -; not taken: 600 x 8192 6.19 / 6.54 / 10.81, 4096 x 2048 9.10 / 9.98 / 9.92.  With a product behind it,
  // 4096 columns, 24 x 4096 10.5 -> 9.0, 300 x 2048 13.2 -> 11.1.
  auto threads_for = [&](int keep) {
    int t = 32;
    while (t < 1024 && chunks > (int64_t)t * keep) t *= 2;
    return t;
  };
  int keep = 4, tpr = 32;
  if (chunks <= 512 && M * threads_for(1) <= 1100ll * sms) keep = 1;
  else if (chunks <= 2048 && M * threads_for(2) <= 1100ll * sms) keep = 2;
  if (keep < 4) {
    tpr = threads_for(keep);
  } else {
    while (tpr < qg::AQ_THREADS && chunks > (int64_t)tpr * 4) tpr *= 2;
    if (chunks > (int64_t)tpr * 4) keep = qg::AQ_MAX_CHUNKS;
  }
  const int block = qg::aq_block(tpr);
  const int64_t rows_per_block = block / tpr;
  const int64_t grid = (M + rows_per_block - 1) / rows_per_block;
  if (grid > 0x7fffffffll) return fail("qgemm_act_quant: too many rows (%lld)", (long long)M);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // A programmatic dependent: behind a W8A8 kernel it is resident when that kernel ends, and behind any other its launch is ready.
  // With more blocks than SMs they first fill the SMs that a GEMM kernel leaves idle in its last round, but in plain stream order the
  // launch costs more.  us, plain / early, calls one after another: by itself 4096 x 4096 16.5 / 14.6, 8192 x 1024 10.3 / 8.5, with the GEMM
  // behind it 600 x 4096 x 4096 22.0 / 20.1, 361 x 2464 x 2768 14.4 / 12.5, but 3000 x 1024 x 1024 15.6 / 16.1, 775 x 3968 x 11056 47.1 / 48.3; 60
  // such pairs of 150 .. 4096 rows 6 % faster in the mean (as one graph, where a plain launch costs less, 1 % slower).
  auto launch = [&](auto kernel) { return launch_pdl(kernel, (int)grid, block, 0, st, p); };
  auto launch_few = [&](auto keep_) {  // one or two chunks per thread
    constexpr int KEEP = decltype(keep_)::value;
    switch (tpr) {
      case 32: return launch(qg::act_quant_kernel<32, KEEP>);
      case 64: return launch(qg::act_quant_kernel<64, KEEP>);
      case 128: return launch(qg::act_quant_kernel<128, KEEP>);
      case 256: return launch(qg::act_quant_kernel<256, KEEP>);
      case 512: return launch(qg::act_quant_kernel<512, KEEP>);
      default: return launch(qg::act_quant_kernel<1024, 2>);
    }
  };
  if (keep == 1) return launch_few(std::integral_constant<int, 1>{});
  if (keep == 2) return launch_few(std::integral_constant<int, 2>{});
  if (keep == qg::AQ_MAX_CHUNKS) return launch(qg::act_quant_kernel<256, qg::AQ_MAX_CHUNKS>);
  switch (tpr) {
    case 32: return launch(qg::act_quant_kernel<32, 4>);
    case 64: return launch(qg::act_quant_kernel<64, 4>);
    case 128: return launch(qg::act_quant_kernel<128, 4>);
    default: return launch(qg::act_quant_kernel<256, 4>);
  }
}

int qgemm_w4a8(const int8_t* A, const uint8_t* qB, int8_t* workspace, void* C, int64_t M, int64_t N, int64_t K,
               int signed_nibbles, int out_dtype, uint32_t* status, void* stream) {
  if (workspace == nullptr) return fail("qgemm_w4a8: the int8 [N, K] workspace must not be null");
  if (K % 32 != 0 || N % 16 != 0) return fail("qgemm_w4a8: K must be a multiple of 32 and N of 16 (got K=%lld, N=%lld)", (long long)K, (long long)N);
  if (out_dtype == QGEMM_DT_I32 && M > 0 && N > 0 && K > 0 && A != nullptr && qB != nullptr && C != nullptr &&
      aligned16(A) && aligned16(qB) && aligned16(C)) {
    const int rc = w4a8_fused(A, qB, workspace, static_cast<int*>(C), M, N, K, signed_nibbles, status,
                              static_cast<cudaStream_t>(stream));
    if (rc <= 0) return rc;
  }
  if (qgemm_unpack_int4(qB, workspace, N, K, signed_nibbles, stream)) return -1;
  if (out_dtype == QGEMM_DT_I32)
    return qgemm_w8a8(A, workspace, nullptr, nullptr, C, nullptr, 1, M, N, K, 1, 0, QGEMM_DT_I32, QGEMM_B_NK, status, stream);
  return fail("qgemm_w4a8: out_dtype must be I32; cast the result on the caller's side (got %d)", out_dtype);
}

int qgemm_w4a8_act_quant(const void* X, int x_dtype, const uint8_t* qB, int8_t* workspace, int32_t* C, float* scale_a,
                         int round_scale, int64_t M, int64_t N, int64_t K, int signed_nibbles, uint32_t* status,
                         void* stream) {
  if (X == nullptr || qB == nullptr || workspace == nullptr || C == nullptr || scale_a == nullptr)
    return fail("qgemm_w4a8_act_quant: X, qB, workspace, C and scale_a must not be null");
  if (x_dtype != QGEMM_DT_F16 && x_dtype != QGEMM_DT_BF16) return fail("qgemm_w4a8_act_quant: x_dtype must be F16 or BF16 (got %d)", x_dtype);
  if (M <= 0 || N <= 0 || K <= 0) return fail("qgemm_w4a8_act_quant: M, N, K must be positive (got %lld, %lld, %lld)", (long long)M, (long long)N, (long long)K);
  if (K % 32 != 0 || N % 16 != 0) return fail("qgemm_w4a8_act_quant: K must be a multiple of 32 and N of 16 (got K=%lld, N=%lld)", (long long)K, (long long)N);
  if (!aligned16(X) || !aligned16(qB) || !aligned16(C) || !aligned16(workspace)) return fail("qgemm_w4a8_act_quant: pointers must be 16-byte aligned");
  if (M > 128)
    return fail("qgemm_w4a8_act_quant: the fused form covers M <= 128 (got %lld); use qgemm_act_quant and qgemm_w4a8 above that", (long long)M);
  const int rc = w4a8_fused(nullptr, qB, workspace, C, M, N, K, signed_nibbles, status, static_cast<cudaStream_t>(stream), X,
                            x_dtype == QGEMM_DT_BF16 ? 1 : 0, round_scale, scale_a);
  if (rc > 0) return fail("qgemm_w4a8_act_quant: the [N, K] workspace is too small for the kernel's scratch (N * K = %lld bytes)", (long long)(N * K));
  return rc;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------------
// Allocation-free W4A16 entry point.
//
// The scratch memory of the W4A16 kernels (split-K arrival counters, fp32 partial sums, the f16 copy
// of the activations) lives here in a device array that is part of the library image, so a caller
// never has to provide or allocate it.  Every GPU that loads the library carries this array until the
// process exits.
// ---------------------------------------------------------------------------------------------------
namespace {

constexpr int64_t kStaticMaxM = QGEMM_W4A16_NOALLOC_MAX_M;
constexpr int64_t kStaticMaxK = QGEMM_W4A16_NOALLOC_MAX_K;
constexpr int64_t kStaticMaxSms = 160;
constexpr int64_t kStaticScratchBytes =
    kW4CounterBytes + kStaticMaxSms * 2 * kStaticMaxM * 128 * 4 + (kStaticMaxK / 128) * qg::w4g_half_bytes(kStaticMaxM);  // about 6.3 MB

static __device__ __align__(256) unsigned char g_w4a16_static_scratch[kStaticScratchBytes];

// Device address of the array above, per device.  In host code the array's name is only a handle for
// the runtime, not a pointer a kernel could use: the real address comes from cudaGetSymbolAddress and
// differs from GPU to GPU.
void* g_static_scratch_addr[kMaxDevices] = {};
std::mutex g_static_mu;

int static_scratch_for_current_device(void** out) {
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return fail("device index %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (g_static_scratch_addr[dev] == nullptr) {
    void* ptr = nullptr;
    CUDA_OK(cudaGetSymbolAddress(&ptr, g_w4a16_static_scratch));
    if (ptr == nullptr) return fail("cudaGetSymbolAddress returned a null address for the static scratch array");
    g_static_scratch_addr[dev] = ptr;
  }
  *out = g_static_scratch_addr[dev];
  return 0;
}

}  // namespace

extern "C" int qgemm_w4a16_noalloc(const void* A, const uint8_t* B_packed, const void* scales, int zero,
                                   int64_t group, void* C, int64_t M, int64_t N, int64_t K, int a_dtype,
                                   int out_dtype, uint32_t* status, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return fail("qgemm_w4a16_noalloc: M, N, K must be positive (got %lld, %lld, %lld)", (long long)M, (long long)N, (long long)K);
  if (M > kStaticMaxM || K > kStaticMaxK)
    return fail("qgemm_w4a16_noalloc: the built-in scratch covers M <= %lld and K <= %lld (got M=%lld, K=%lld); "
                "use qgemm_w4a16 with a caller-provided workspace for larger problems",
                (long long)kStaticMaxM, (long long)kStaticMaxK, (long long)M, (long long)K);
  const int64_t need = qgemm_w4a16_workspace_bytes(M, N, K);
  if (need < 0) return -1;
  if (need > kStaticScratchBytes)
    return fail("qgemm_w4a16_noalloc: this problem needs %lld bytes of scratch on this device, the built-in array has %lld",
                (long long)need, (long long)kStaticScratchBytes);
  void* scratch = nullptr;
  if (static_scratch_for_current_device(&scratch)) return -1;
  // The array keeps whatever the previous call left behind.  The arrival counters must start at zero: the
  // pre-pass kernel of every call zeroes them; everything else is written before it is read.  Nothing is put
  // on the stream before qgemm_w4a16 has validated the remaining arguments.
  return qgemm_w4a16(A, B_packed, scales, zero, group, C, scratch, kStaticScratchBytes, M, N, K, a_dtype, out_dtype,
                     status, stream);
}
