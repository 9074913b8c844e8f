// C ABI of the chunked XMC classifier layer (see include/elmo_xmc.h): handle, workspaces, TMA
// descriptors and the per-step launch schedule.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "../../include/elmo_xmc.h"
#include "aux_kernels.cuh"
#include "gemm_engine.cuh"
#include "gradx_kernel.cuh"
#include "slim_step.cuh"
#include "xmc_policies.cuh"

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

#define CU_TRY(expr)                                                                         \
  do {                                                                                       \
    cudaError_t e_ = (expr);                                                                 \
    if (e_ != cudaSuccess)                                                                   \
      return fail(XMC_ERR_CUDA, "%s failed: %s (%s:%d)", #expr, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

int get_encode(EncodeFn* out) {
  static EncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    CU_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (p == nullptr || q != cudaDriverEntryPointSuccess)
      return fail(XMC_ERR_CUDA, "cuTensorMapEncodeTiled is not available in this driver");
    fn = reinterpret_cast<EncodeFn>(p);
  }
  *out = fn;
  return XMC_OK;
}

// Encoding a tensor map costs a few microseconds on the host and a step needs ~26 of them with
// arguments that repeat every step, so encoded maps are remembered (per thread, direct-mapped).
struct MapKey {
  uint64_t base, a, b, c;
  uint32_t kind, e4m3, box0, box1, swizzle, pad;
  bool operator==(const MapKey& o) const { return memcmp(this, &o, sizeof(MapKey)) == 0; }
};
struct MapSlot {
  MapKey key;
  CUtensorMap map;
  bool used = false;
};
constexpr int kMapSlots = 512;
inline MapSlot* map_slot(const MapKey& k) {
  static thread_local MapSlot slots[kMapSlots];
  uint64_t h = k.base * 0x9E3779B97F4A7C15ull ^ (k.a * 0xC2B2AE3D27D4EB4Full) ^ (k.b << 17) ^ (k.c << 3) ^
               ((uint64_t)k.kind << 60) ^ ((uint64_t)k.box1 << 40) ^ ((uint64_t)k.box0 << 50) ^ k.e4m3 ^ ((uint64_t)k.swizzle << 1);
  h ^= h >> 29;
  return &slots[h % kMapSlots];
}

// 2-D row-major tensor [outer x inner], box [box_outer x box_inner], zero fill.
enum { SWIZZLE_NONE = 0, SWIZZLE_128 = 1, SWIZZLE_64 = 2 };
int make_map(CUtensorMap* m, bool e4m3, const void* base, uint64_t inner, uint64_t outer,
             uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, uint32_t swizzle = SWIZZLE_128) {
  EncodeFn enc;
  if (int rc = get_encode(&enc)) return rc;
  if (((uintptr_t)base & 15u) != 0 || (row_stride_bytes & 15u) != 0)
    return fail(XMC_ERR_INVALID, "tensor base/stride must be 16-byte aligned (base %p, stride %llu)", base,
                (unsigned long long)row_stride_bytes);
  MapKey key;
  memset(&key, 0, sizeof(key));
  key.base = (uint64_t)(uintptr_t)base; key.a = inner; key.b = outer; key.c = row_stride_bytes;
  key.kind = 2; key.e4m3 = e4m3; key.box0 = box_inner; key.box1 = box_outer; key.swizzle = swizzle;
  MapSlot* slot = map_slot(key);
  if (slot->used && slot->key == key) {
    *m = slot->map;
    return XMC_OK;
  }
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {row_stride_bytes};
  const cuuint32_t box[2] = {box_inner, box_outer};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = enc(m, e4m3 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swizzle == SWIZZLE_128 ? CU_TENSOR_MAP_SWIZZLE_128B : swizzle == SWIZZLE_64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(XMC_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d): inner %llu outer %llu stride %llu box %ux%u",
                (int)r, (unsigned long long)inner, (unsigned long long)outer,
                (unsigned long long)row_stride_bytes, box_inner, box_outer);
  slot->key = key;
  slot->map = *m;
  slot->used = true;
  return XMC_OK;
}
// [rows x cols] row-major matrix seen as [cols/64 blocks][rows][64 elements]: one box fetches
// `box_rows` rows of `box_blocks` consecutive 64-element blocks, laid out block after block in shared memory
// (each block = box_rows rows of 64 elements).  Blocks/rows outside the matrix read as zero.
int make_map_blocked(CUtensorMap* m, bool e4m3, const void* base, uint64_t cols, uint64_t rows,
                     uint64_t row_stride_elems, uint32_t box_rows, bool swizzle, uint32_t box_blocks = 4) {
  EncodeFn enc;
  if (int rc = get_encode(&enc)) return rc;
  const uint32_t es = e4m3 ? 1 : 2;
  if (cols % 64 != 0) return fail(XMC_ERR_INVALID, "blocked tensor map needs a multiple of 64 columns, got %llu", (unsigned long long)cols);
  if (((uintptr_t)base & 15u) != 0 || ((row_stride_elems * es) & 15u) != 0)
    return fail(XMC_ERR_INVALID, "tensor base/stride must be 16-byte aligned");
  MapKey key;
  memset(&key, 0, sizeof(key));
  key.base = (uint64_t)(uintptr_t)base; key.a = cols; key.b = rows; key.c = row_stride_elems;
  key.kind = 3; key.e4m3 = e4m3; key.box0 = 64; key.box1 = box_rows; key.swizzle = swizzle; key.pad = box_blocks;
  MapSlot* slot = map_slot(key);
  if (slot->used && slot->key == key) {
    *m = slot->map;
    return XMC_OK;
  }
  const cuuint64_t dims[3] = {64, rows, cols / 64};
  const cuuint64_t strides[2] = {row_stride_elems * es, 64ull * es};
  const cuuint32_t box[3] = {64, box_rows, box_blocks};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(m, e4m3 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3,
                         const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(XMC_ERR_CUDA, "cuTensorMapEncodeTiled (blocked) failed (%d): cols %llu rows %llu stride %llu",
                (int)r, (unsigned long long)cols, (unsigned long long)rows, (unsigned long long)row_stride_elems);
  slot->key = key;
  slot->map = *m;
  slot->used = true;
  return XMC_OK;
}
// operand whose K runs along the rows' contiguous direction
int make_map_kmajor(CUtensorMap* m, bool e4m3, const void* base, uint64_t k_elems, uint64_t rows,
                    uint64_t row_stride_elems, uint32_t box_rows) {
  const uint32_t es = e4m3 ? 1 : 2;
  return make_map(m, e4m3, base, k_elems, rows, row_stride_elems * es, 128 / es, box_rows);
}
// e4m3 rows [rows x k_bytes] fetched raw, 64 bytes (one bf16 k-step) of `box_rows` rows per box, for the
// in-kernel conversion to a bf16 operand
int make_map_raw8(CUtensorMap* m, const void* base, uint64_t k_bytes, uint64_t rows, uint64_t row_stride_bytes,
                  uint32_t box_rows) {
  return make_map(m, true, base, k_bytes, rows, row_stride_bytes, 64, box_rows, SWIZZLE_NONE);
}
// bf16 operand stored [k_rows x mn] (MN contiguous): boxes of box_rows k-rows x 64 elements
int make_map_mnmajor(CUtensorMap* m, const void* base, uint64_t mn, uint64_t k_rows,
                     uint64_t row_stride_elems, uint32_t box_rows = 64) {
  return make_map(m, false, base, mn, k_rows, row_stride_elems * 2, 64, box_rows);
}

// Launch with programmatic stream serialization: the kernel may be scheduled while its predecessor in
// the stream drains; it orders itself with griddepcontrol.wait before its first global access.
// cluster > 1 launches thread-block clusters of that many CTAs along x.
inline void launch_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at, int grid, int block, size_t smem,
                          cudaStream_t stream, int cluster) {
  memset(cfg, 0, sizeof(*cfg));
  cfg->gridDim = dim3((unsigned)grid);
  cfg->blockDim = dim3((unsigned)block);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = stream;
  static const bool no_pdl = getenv("XMC_NO_PDL") != nullptr;
  int n = 0;
  if (!no_pdl) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = (unsigned)cluster;
    at[n].val.clusterDim.y = 1;
    at[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg->attrs = at;
  cfg->numAttrs = n;
}
template <class Kern, class... Args>
cudaError_t launch_pdl(Kern kern, int grid, int block, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  launch_config(&cfg, at, grid, block, smem, stream, 1);
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// dynamic shared memory opt-in of the grad_X kernels, once per device; *max_pairs = CTA pairs of the pair
// kernel the device holds at once
int gradx_configure(int sm_count, int* max_pairs) {
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> pairs[64];
  int dev = 0;
  CU_TRY(cudaGetDevice(&dev));
  if (!((configured.load(std::memory_order_acquire) >> (dev & 63)) & 1ull)) {
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<true, false, 2>));
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<false, false, 2>));
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<true, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<true, true, 1>));
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<true, true, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<true, true, 2>));
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<false, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<false, true, 1>));
    // every pair kernel has an SM to itself: they fit the same number of times
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    launch_config(&cfg, at, sm_count / 2 * 2, xmc::kGxThreads, xmc::kGxSmemBytes<true, true, 2>, nullptr, 2);
    int n = 0;
    CU_TRY(cudaOccupancyMaxActiveClusters(&n, xmc::gradx_kernel<true, true, 2>, &cfg));
    pairs[dev & 63].store(std::max(0, std::min(n, sm_count / 2)), std::memory_order_relaxed);
    configured.fetch_or(1ull << (dev & 63), std::memory_order_release);
  }
  *max_pairs = pairs[dev & 63].load(std::memory_order_relaxed);
  return XMC_OK;
}

// the parts of the update's parameters that one step shares: random stream and learning rate
void fill_update_stream(xmc::UpdParams* up, uint64_t seed, uint64_t step, float lr_eff, float wd) {
  up->lr_eff = lr_eff;
  up->wd = wd;
  up->seed = seed;
  up->step = step;
  for (int rd = 0; rd < xmc::kSrRounds; ++rd) {
    up->rkey[rd][0] = (uint32_t)seed + (uint32_t)rd * 0x9E3779B9u;
    up->rkey[rd][1] = (uint32_t)(seed >> 32) + (uint32_t)rd * 0xBB67AE85u;
  }
  const unsigned long long m = 0xCD9E8D57ull * (uint32_t)step;
  up->sr_x1 = (uint32_t)(m >> 32) ^ up->rkey[0][0];
  up->sr_y1 = (uint32_t)m ^ up->rkey[1][0];
  up->sr_z1 = (uint32_t)(step >> 32) ^ up->rkey[0][1];
}

// Launch of the one-kernel step; *grid_out = CTAs launched (two per cluster).
template <bool W8, bool SR, bool LOSS, xmc::KahanTerms KAHAN, bool U_WAITS, bool SPLIT = false, bool BOUND = false>
int launch_slim(const CUtensorMap& x, const CUtensorMap& xt, const xmc::SlimParams& p, int smem, int max_clusters, int sm_count,
                cudaStream_t stream, int* grid_out) {
  auto kern = xmc::slim_step_kernel<W8, SR, LOSS, KAHAN, U_WAITS, SPLIT, BOUND>;
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> clusters[64];
  int dev = 0;
  CU_TRY(cudaGetDevice(&dev));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  if (!((configured.load(std::memory_order_acquire) >> (dev & 63)) & 1ull)) {
    CU_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
    launch_config(&cfg, at, sm_count / 2 * 2, xmc::kSlThreads, 232448, stream, 2);
    int n = 0;
    CU_TRY(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
    if (n <= 0) return fail(XMC_ERR_CUDA, "the device cannot hold a pair of CTAs of this kernel");
    // the warpgroups share out exactly these
    cudaFuncAttributes attr;
    CU_TRY(cudaFuncGetAttributes(&attr, kern));
    if (attr.numRegs != xmc::kSlLaunchRegs)
      return fail(XMC_ERR_CUDA, "the one-kernel step was compiled for %d registers a thread, not %d", attr.numRegs, xmc::kSlLaunchRegs);
    clusters[dev & 63].store(std::min(n, sm_count / 2), std::memory_order_relaxed);
    configured.fetch_or(1ull << (dev & 63), std::memory_order_release);
  }
  const int grid = 2 * std::min(std::min(p.n_tiles, max_clusters), clusters[dev & 63].load(std::memory_order_relaxed));
  *grid_out = grid;
  launch_config(&cfg, at, grid, xmc::kSlThreads, smem, stream, 2);
  CU_TRY(cudaLaunchKernelEx(&cfg, kern, x, xt, p));
  return XMC_OK;
}

// PAIR: the kernel runs on CTA pairs (clusters of two); n_tiles then counts the pairs' 256-row tiles and
// the grid is twice the number of pairs the device can hold at once (asked of the occupancy calculator:
// an SM that has no partner within its GPC cannot take part).
template <class Policy, bool PAIR = false>
int launch_gemm(const CUtensorMap& a, const CUtensorMap& b, const typename Policy::Params& p, int n_tiles,
                int sm_count, cudaStream_t stream, int grid_override = 0, const CUtensorMap* c = nullptr,
                int* grid_out = nullptr) {
  if (n_tiles <= 0) return XMC_OK;
  auto kern = xmc::gemm_kernel<Policy, PAIR>;
  constexpr int smem = xmc::smem_bytes<Policy, PAIR>();
  constexpr int block = xmc::block_threads<Policy>();
  // once per device and kernel (one process may drive several devices)
  static std::atomic<uint64_t> configured{0};
  static std::atomic<int> max_pairs[64];
  int dev = 0;
  CU_TRY(cudaGetDevice(&dev));
  if (!((configured.load(std::memory_order_acquire) >> (dev & 63)) & 1ull)) {
    CU_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (PAIR) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute at[2];
      launch_config(&cfg, at, sm_count / 2 * 2, block, smem, stream, 2);
      int n = 0;
      CU_TRY(cudaOccupancyMaxActiveClusters(&n, kern, &cfg));
      if (n <= 0) return fail(XMC_ERR_CUDA, "the device cannot hold a pair of CTAs of this kernel");
      max_pairs[dev & 63].store(std::min(n, sm_count / 2), std::memory_order_relaxed);
    }
    configured.fetch_or(1ull << (dev & 63), std::memory_order_release);
  }
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  int grid;
  if (PAIR) grid = 2 * (grid_override > 0 ? grid_override : std::min(n_tiles, max_pairs[dev & 63].load(std::memory_order_relaxed)));
  else grid = grid_override > 0 ? grid_override : std::min(n_tiles, sm_count);
  if (grid_out != nullptr) *grid_out = grid;
  launch_config(&cfg, at, grid, block, smem, stream, PAIR ? 2 : 1);
  CU_TRY(cudaLaunchKernelEx(&cfg, kern, a, b, c ? *c : a, p));
  return XMC_OK;
}

// Label rows whose contribution to grad_X one TMEM accumulator sums up before it is added to the fp32 partial sums in
// memory.  The tensor core truncates where it adds to an accumulator, so the error grows with the length of the sum:
// bf16 weights U(+-1/sqrt(d)), relative 2-norm error of the fp32 grad_X against 64 bits, unbounded and with these bounds:
// 131 072 x 768 batch 256 1.8e-6 and 3.1e-7, 500 000 x 256 batch 140 8.9e-7 and 2.0e-7, one-kernel step 300 000 x 768 batch 128
// 3.1e-6 and 2.1e-7, 2 000 000 x 64 batch 8 1.4e-5 and 3.1e-7.  The bounds are what a launch of 32 768 rows gives each
// split, but not below 512: shorter sums cost time on single CTAs (300 000 x 768 in the one-kernel step at 128 345 -> 395;
// with 256 rows 455) and gain nothing on the fp32 additions.  On pairs they are always 512: the sums there grow in
// registers.  e4m3 weights are not bounded within a launch of the three kernels: a product has 12 significant bits, and the same weights as
// e4m3 sum up to within 4e-8 to 7e-8 as long as a sum stays below 2^24 of its smallest bits -- with 64 features, whose weights are
// the largest, no longer than that (slim_sum_tiles).  Stored weights spread evenly over ten binades need more, and there the
// length shows: 670 091 x 768 at batch 32 (one kernel) 6.0e-6, 140 2.1e-6, 256 4.2e-6, 512 1.8e-6.
constexpr int kChainRows = 32768, kMinChainRows = 512;
constexpr int kSlimChainTiles = kMinChainRows / 128;     // a power of two

inline int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }
inline long long round_up(long long a, long long b) { return (a + b - 1) / b * b; }

}  // namespace

struct xmc_handle {
  xmc_config cfg{};
  int sm_count = 0;
  int bpad_max = 0;
  int tile_rows = 0;               // label rows of a tile: 256 (CTA pairs) or 128
  int tiles_per_chunk = 0, n_tiles = 0;   // label tiles of a weight chunk (padded to whole ones), of all chunks
  int launch_tiles = 0;            // label tiles per launch of the step's kernels
  int64_t g_rows = 0;              // rows of G currently allocated: launch_tiles * tile_rows
  std::vector<void*> w_ptrs;
  std::vector<int64_t> w_rows;
  int64_t total_rows = 0;
  int64_t rows_per_chunk = 0;
  int n_buckets = 0;
  int64_t w_maps_bytes = 0;
  CUtensorMap* w_maps = nullptr;   // device array [W_MAPS][chunks] of tensor maps (enum below)
  // workspaces; x8, x16, xt, partial and status are parts of the arena
  void* arena = nullptr;
  uint8_t* x8 = nullptr;           // [max(bpad_max,256) x d] e4m3; simulated FP8: the parts of split embeddings, PrepX::parts
  __nv_bfloat16* x16 = nullptr;    // [max(bpad_max,256) x d]
  float* x_scale = nullptr;        // [max(bpad_max,256)] simulated FP8
  uint8_t* x_wide = nullptr;       // [max(bpad_max,256)] simulated FP8; zero at first, like the parts
  __nv_bfloat16* xt = nullptr;     // [max(d,256) x bpad_max]
  __nv_bfloat16* G = nullptr;      // [sched x bpad_max]
  uint8_t* G8 = nullptr;           // [sched x bpad_max] e4m3(G * 256), allocated when the FP8 dW contraction is first asked for
  uint8_t* xt8 = nullptr;          // [max(d,256) x bpad_max] e4m3 X transposed, likewise
  int64_t g8_rows = 0;
  float* partial = nullptr;
  int64_t partial_floats = 0;
  int* bucket_cnt = nullptr;       // [2 * n_buckets] counts then cursors
  int* bucket_off = nullptr;       // [n_buckets + 1]
  uint32_t* entries = nullptr;
  int64_t ent_cap = 0;
  double* loss_partial = nullptr;
  int64_t loss_cap = 0;
  int* status = nullptr;           // 4 ints
  unsigned long long* stats = nullptr;   // weight statistics: 4 counters + the largest magnitude byte
  int64_t ws_bytes = 0;
  // bookkeeping for the bench: kernels launched so far, optional per-kernel-class event timing
  // fused top-k: per 32 labels of a window the largest logit, and per batch row the best so far (grown on demand)
  uint16_t* topk_gmax = nullptr;
  int64_t topk_gmax_cap = 0;       // entries
  unsigned long long* topk_run = nullptr;
  int* topk_cnt = nullptr;
  float* topk_thr = nullptr;
  void* kahan = nullptr;           // borrowed compensation buffer for the first kahan_rows rows
  int64_t kahan_rows = 0;
  int kahan_e5m2 = 0;
  int64_t l2_persist_bytes = 0;    // size of the persisting-L2 carve-out this process asked for (0 = none)
  int64_t launches = 0;
  bool profile = false;
  std::vector<cudaEvent_t> ev_pool;
  std::vector<int> ev_kind;        // kind of the kernel that FOLLOWS event i
  size_t ev_used = 0;
};

// Tensor maps of the weight chunks, kept in device memory: a launch covers tiles of several chunks.
enum {
  W_ROWS128 = 0,   // boxes of 128 rows x 128 bytes, 128-byte swizzle: operand as stored, the update's weight block
  W_ROWS256,       // the same of 256 rows (single-CTA logits and top-k)
  W_RAW128,        // simulated FP8: 64 bytes of 128 / 256 rows, unswizzled, for the conversion in the kernel
  W_RAW256,
  W_GX2,           // grad_X: 64-element blocks of kGxRows rows, two (CTA pairs) or four of them
  W_GX4,
  W_MAPS
};

namespace {

// What the legacy stream has been given -- zero fills, and copies from pageable memory, which may return before the data
// has arrived -- is done: the caller's stream need not wait for that stream (torch's side streams do not).
int host_work_done() {
  CU_TRY(cudaStreamSynchronize(cudaStreamLegacy));
  return XMC_OK;
}

int dev_alloc(xmc_handle* h, void** p, size_t bytes, bool zero) {
  if (const cudaError_t e = cudaMalloc(p, bytes)) {
    *p = nullptr;
    cudaGetLastError();                    // not for the next call to find
    return fail(XMC_ERR_CUDA, "allocating %zu bytes failed: %s", bytes, cudaGetErrorString(e));
  }
  if (zero) {
    CU_TRY(cudaMemsetAsync(*p, 0, bytes, cudaStreamLegacy));
    if (int rc = host_work_done()) return rc;
  }
  h->ws_bytes += (int64_t)bytes;
  return XMC_OK;
}

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

// Count a kernel launch; in profile mode also drop an event in front of it.
enum { K_PREP = 0, K_UNUSED = 1, K_FWD = 2, K_GRADX = 3, K_UPD = 4, K_REDUCE = 5, K_LOGITS = 6, K_END = 7 };
void mark(xmc_handle* h, int kind, cudaStream_t st) {
  if (kind != K_END) ++h->launches;
  if (!h->profile) return;
  if (h->ev_used == h->ev_pool.size()) {
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) return;
    h->ev_pool.push_back(e);
    h->ev_kind.push_back(kind);
  }
  h->ev_kind[h->ev_used] = kind;
  cudaEventRecord(h->ev_pool[h->ev_used], st);
  ++h->ev_used;
}

xmc::BucketGeom geom_of(const xmc_handle* h) {
  xmc::BucketGeom g;
  g.label_offset = h->cfg.label_offset;
  g.total_rows = h->total_rows;
  g.rows_per_chunk = (int)h->rows_per_chunk;
  g.per_chunk = cdiv(h->rows_per_chunk, 128);
  g.n_buckets = h->n_buckets;
  return g;
}
const CUtensorMap* chunk_maps(const xmc_handle* h, int kind) { return h->w_maps + (size_t)kind * h->w_ptrs.size(); }
// tiles [first, first + count) of m_rows label rows each
xmc::LabelTiles label_tiles(const xmc_handle* h, int m_rows, int first, int count) {
  xmc::LabelTiles t;
  t.m_rows = m_rows;
  const int per = cdiv(h->rows_per_chunk, m_rows);
  t.per_chunk = xmc::make_fastdiv(per, (long long)per * (long long)h->w_ptrs.size());
  t.rows_full = (int)h->rows_per_chunk;
  t.rows_last = (int)h->w_rows.back();
  t.n_chunks = (int)h->w_ptrs.size();
  t.first = first;
  t.count = count;
  return t;
}
// label tiles of 256 that hold the handle's rows [0, n)
int tiles_up_to(const xmc_handle* h, int64_t n) {
  const int64_t chunk = (n - 1) / h->rows_per_chunk;
  return (int)(chunk * cdiv(h->rows_per_chunk, 256) + (n - 1 - chunk * h->rows_per_chunk) / 256 + 1);
}
bool use_pairs(int max_pairs) {
  static const bool no_pairs = getenv("XMC_NO_PAIRS") != nullptr;
  return !no_pairs && max_pairs >= 1;
}

int x_rows_of(const xmc_handle* h) { return std::max(h->bpad_max, 256); }     // rows of the embeddings' arrays
// split embeddings as an operand: the parts, one below the other
int make_map_parts(xmc_handle* h, CUtensorMap* map, int box_rows) {
  return make_map_kmajor(map, true, h->x8, h->cfg.dim, 4 * (size_t)x_rows_of(h), h->cfg.dim, (uint32_t)box_rows);
}
xmc::PrepX prep_args(xmc_handle* h, const void* x, int x_dtype, int batch, int bpad, bool need_x8, bool need_x16, bool need_xt, bool need_xt8,
                     bool split, int* blocks) {
  xmc::PrepX p;
  p.x = x;
  p.batch = batch;
  p.bpad = bpad;
  p.d = h->cfg.dim;
  p.row_blocks = split && x_dtype != XMC_DT_E4M3 ? cdiv(bpad, xmc::kSplitRows) : 0;
  p.x8 = need_x8 || (split && p.row_blocks == 0) ? h->x8 : nullptr;
  p.x16 = need_x16 ? h->x16 : nullptr;
  p.xt = need_xt ? h->xt : nullptr;
  p.xt8 = need_xt8 ? h->xt8 : nullptr;
  p.parts = split ? h->x8 : nullptr;
  p.part_bytes = (size_t)x_rows_of(h) * p.d;
  p.x_wide = h->x_wide;
  p.x_scale = h->x_scale;
  p.w_scale = h->cfg.w_scale;
  *blocks = p.row_blocks;
  if (p.x8 != nullptr || need_x16 || need_xt || need_xt8) *blocks += cdiv(p.d, 32) * cdiv(bpad, 32);
  return p;
}
int prep_x(xmc_handle* h, const void* x, int x_dtype, int batch, int bpad, bool need_x8, bool need_x16, bool need_xt,
           cudaStream_t st, bool need_xt8 = false, bool split = false, int early = 0) {
  int blocks;
  const xmc::PrepX p = prep_args(h, x, x_dtype, batch, bpad, need_x8, need_x16, need_xt, need_xt8, split, &blocks);
  mark(h, K_PREP, st);
  CU_TRY(x_dtype == XMC_DT_E4M3 ? launch_pdl(xmc::prep_x_kernel<true, false>, blocks, xmc::kPrepThreads, 0, st, p, early)
                                : launch_pdl(p.row_blocks > 0 ? xmc::prep_x_kernel<false, true> : xmc::prep_x_kernel<false, false>, blocks, xmc::kPrepThreads, 0, st, p, early));
  return XMC_OK;
}
// The embeddings of an inference call as the kernels' operand.  Where they come in the operand's own type they are read
// in place -- rows beyond the batch lie outside of the map and read as zero -- and the call is one launch shorter: a
// small one is bound by the host, 2 us a launch, and waits 4 us less on the GPU.  A training step has to prepare
// X^T anyway.  A map wants a 16-byte aligned address.
// Else *own_prep, up to batch 128: the kernel behind may start as soon as all before the preparation is complete, and fetch
// weights meanwhile (only X has to wait; a merge or nothing follows that kernel, and both wait for it).  Top 5 of 131 072 x 768 for
// one query 23.7 -> 22.2 us, its logits 19.9 -> 18.2; for 300 rows, whose preparation fills the SMs, 60.3 -> 62.6.  (split: make_map_parts.)
int inference_operand(xmc_handle* h, const void* x, int x_dtype, int batch, bool split, int x_rows, CUtensorMap* map, int* own_prep, cudaStream_t st) {
  const int d = h->cfg.dim;
  const bool e4m3 = h->cfg.mode == XMC_MODE_FP8;
  *own_prep = 0;
  if (!split && (x_dtype == XMC_DT_E4M3) == e4m3 && ((uintptr_t)x & 15u) == 0)
    return make_map_kmajor(map, e4m3, x, d, batch, d, (uint32_t)x_rows);
  *own_prep = batch <= 128;
  if (int rc = prep_x(h, x, x_dtype, batch, (int)round_up(batch, 64), e4m3, !e4m3 && !split, false, st, false, split, *own_prep)) return rc;
  const size_t xrows = (size_t)x_rows_of(h);
  if (split) return make_map_parts(h, map, x_rows);
  return make_map_kmajor(map, e4m3, e4m3 ? (const void*)h->x8 : (const void*)h->x16, d, xrows, d, (uint32_t)x_rows);
}
// Rows of a box of embeddings: the batch, in whole groups of eight, where a tile of 128 has more.  (Boxes of 128 rows took a third of what
// the kernel fetches, and where they lie mostly outside of the tensor longer than if they were
// there.  131 072 x 768, us: top 5 for one e4m3 query 25.8 -> 20.0, bf16 weights 47.2 -> 39.6; logits of 7 rows 25.3 -> 20.4, bf16 49.2 -> 36.2.)
int inference_rows(int batch) { return std::min(128, (int)round_up(batch, 8)); }
// Simulated FP8 inference: whether the embeddings are split for the FP8 tensor cores or the weights converted in the kernel.  The split
// halves what a k-step costs (about 500 cycles for 64 features where converting takes 1000) and costs a preparation, 2 to 4 us,
// where the embeddings are read in place otherwise, more of which is hidden up to batch 128; narrow layers fill half of its k-steps
// of 128 features.  Logits converted and split, us: 60 000 x 768 at batch 1 22.9 and 14.1, 131 072 x 768 47.7 and 23.2, at 100 42.8 and 29.0;
// on pairs 30 000 x 768 at 160 (24) 19.3 and 19.8, at 300 (48) 28.9 and 27.1, 100 000 x 256 at 160 (24) 17.3 and 19.7, at 300 (44) 30.6 and
// 30.3, 300 000 x 384 at 300 116 and 92; 500 000 x 128 at 160 62.9 and 67.0, 1 000 000 x 64 at 64 50.7 and 67.1.
bool split_pays(const xmc_handle* h, int tiles, int max_pairs, bool pair) {
  return h->cfg.dim >= 256 && (int64_t)cdiv(tiles, pair ? max_pairs : h->sm_count) * (h->cfg.dim / 64) >= (pair ? 48 : 16);
}

// Shape of the one-kernel step for this batch and feature count, or false where it does not fit: the grad_X
// accumulators of half the features, half a Z and the two teams' update chunks have to share 512 TMEM columns
// (batch 128: up to 768 features, 96: 1 024, 64: 1 536, 32: 3 328), rings and boxes 227 KB (a box of bf16 weights is 32 KB).
bool slim_geometry(bool w8, bool split, bool kahan, bool loss, int batch, int d, xmc::SlimParams* p, int* smem) {
  if (batch > 128) return false;
  p->nb = (int)round_up(batch, 32);
  p->n_boxes = cdiv(d, 128);
  const int cols = ((p->n_boxes + 1) / 2) * p->nb + p->nb / 2;
  // Up to `boxes` boxes of features a row: features per chunk and team, chunks in TMEM, Z stages, weight slots, X^T
  // stages, buffers for G and for copies of e4m3 weights; the first that fits.  Found by trying all that fit, 64 to 1 024 features, batch 8 to 128; times relative to
  // the best of them.  A box a CTA: its X^T stays and G gets the third buffer, as gx(i) lies between G(i) and G(i + 2) (600 000 x 256,
  // batch 8: two buffers 1.05, rounded to nearest 1.15).  e4m3 with more boxes: a third weight slot is worth a stage of Z (300 000 x
  // 768 rounded to nearest, batch 64: two slots 1.11).  bf16, twice the boxes for Z: four stages (200 000 x 512, batch 8: three 1.08), but
  // X^T of two boxes kept where there are three (1.04), and of four boxes one update chunk (512 features, batch 16: two 1.09), but two with
  // the loss, whose G takes longer (batch 40: one 1.07).  bf16 beyond
  // batch 64, where not all of that fits: a row of six boxes and more keeps three stages of Z and takes chunks of 32 features (200 000 x 768 at 80
  // 257 -> 240 us, at 96 rounded to nearest 252 -> 230), shorter ones keep the wider chunks (250 000 x 640 at 80 250, with narrow ones 276), three to five boxes one of
  // them, which leaves TMEM for a second Z.  e4m3 beyond batch 64: one buffer for copies -- the workers need it only when they
  // have a box's first results, by when the box before has been multiplied -- so that X^T has whole boxes or more stages (150 000 x
  // 768 at batch 128 150.0 -> 142.9 us, rounded to nearest 136.9 -> 114.9; 200 000 x 384 at 96 133.5 -> 117.3, 114.7 -> 96.9).  With compensated
  // rows, whose boxes take longer, that pays for whole boxes of X^T only (312 330 x 768 at 128 341 with two buffers, 348 with one; 300 000 x
  // 384 at 96 235 and 219).
  struct Shape { int boxes, uw, u_bufs, z_stages, w_slots, xt_stages, g_bufs, s_bufs; bool loss = false; };     // loss: with the loss only
  static constexpr Shape e4m3[] = {{2, 64, 2, 3, 2, 1, 3, 2}, {2, 64, 2, 2, 2, 1, 3, 2}, {99, 64, 2, 2, 3, 2, 2, 2}, {99, 32, 2, 3, 3, 2, 2, 2}, {99, 32, 2, 2, 3, 2, 2, 2},
                               {99, 64, 2, 2, 2, 1, 2, 1}, {99, 64, 1, 2, 3, 1, 2, 1}, {99, 64, 1, 2, 2, 1, 2, 1}, {99, 32, 1, 2, 3, 2, 2, 1}, {99, 32, 1, 2, 2, 2, 2, 1}, {99, 32, 1, 2, 2, 1, 2, 2}};
  static constexpr Shape bf16[] = {{2, 64, 2, 4, 3, 1, 2, 2}, {3, 64, 2, 3, 3, 2, 2, 2}, {4, 64, 2, 3, 3, 2, 2, 2, true}, {4, 64, 1, 4, 3, 1, 2, 2}, {99, 64, 2, 4, 3, 1, 2, 2}, {99, 32, 2, 4, 3, 2, 2, 2},
                               {2, 64, 2, 2, 2, 1, 2, 2}, {5, 64, 1, 2, 2, 1, 2, 2}, {5, 32, 1, 2, 2, 2, 2, 2},
                               {99, 32, 2, 3, 2, 1, 2, 2}, {99, 32, 1, 3, 2, 1, 2, 2}};
  constexpr auto in_barriers = [](const Shape& t) {          // the barrier arrays have room for no more
    return t.u_bufs <= 2 && t.z_stages <= xmc::kSlMaxZ && t.w_slots <= xmc::kSlMaxW && t.xt_stages <= xmc::kSlMaxXt && t.g_bufs <= xmc::kSlMaxG && t.s_bufs <= xmc::kSlStaging;
  };
  static_assert([=] {
    for (const Shape& t : e4m3) if (!in_barriers(t)) return false;
    for (const Shape& t : bf16) if (!in_barriers(t)) return false;
    return true;
  }());
  const Shape* shapes = w8 ? e4m3 : bf16;
  const int n_shapes = w8 ? (int)(sizeof(e4m3) / sizeof(Shape)) : (int)(sizeof(bf16) / sizeof(Shape));
  for (int i = 0; i < n_shapes; ++i) {
    const Shape& t = shapes[i];
    if (p->n_boxes > t.boxes || (kahan && t.uw == 32 && t.s_bufs == 1) || (t.loss && !loss)) continue;
    p->uw = t.uw;
    p->u_bufs = t.u_bufs;
    p->z_stages = t.z_stages;
    p->w_slots = t.w_slots;
    p->xt_stages = t.xt_stages;
    p->g_bufs = t.g_bufs;
    p->s_bufs = t.s_bufs;
    *smem = xmc::slim_smem_bytes(w8, split, p->nb, t.uw, t.z_stages, t.w_slots, t.xt_stages, t.g_bufs, t.s_bufs);
    const int u_cols = t.u_bufs * 2 * t.uw;
    p->z_bufs = cols + p->nb / 2 + u_cols <= 512 ? 2 : 1;        // with a second Z the next contraction goes on while the first one waits for G
    if (cols + u_cols <= 512 && *smem <= 232448) return true;
  }
  return false;
}

// Splits of grad_X on single CTAs, a CTA for each of n_bt x n_dt tiles and split.
int gx_splits(const xmc_handle* h, int workers, int n_bt, int n_dt, int bpad) {
  int n = std::max(1, workers / (n_bt * n_dt));
  while (n > 1 && (int64_t)n * bpad * h->cfg.dim > h->partial_floats) --n;
  return n;
}
int slim_tiles(const xmc_handle* h) { return (int)(h->w_ptrs.size() - 1) * cdiv(h->rows_per_chunk, 128) + cdiv(h->w_rows.back(), 128); }

// Label tiles of 128 that a grad_X accumulator of the one-kernel step sums up over e4m3 weights at most, where the kernel can end a sum
// (BOUND): as many as in the three kernels, a launch over its splits, or 32.  Real FP8 up to half as many rows as features never had
// other sums and is not bounded.  Relative error against 64 bits, three kernels, one kernel unbounded and as it is, weights
// U(+-1/sqrt(d)): FP8 rounded to nearest 1 000 000 x 64 at batch 128 5.1e-8, 1.2e-6 and 6.0e-8, 2 800 000 x 64 3.9e-8, 2.9e-5 and 4.8e-8, 1 000 000
// x 192 5.2e-8, 4.9e-8 and 4.9e-8; weights over ten binades: the first two 4.1e-7, 8.5e-6 and 2.4e-6, and 6.6e-7, 1.2e-5 and 2.6e-6 (their
// launches are short), simulated FP8 2 812 281 x 768 at 128 7.6e-6, 1.2e-5 and 7.1e-6, at 16 8.5e-6, 1.2e-5 and 8.5e-6.
int slim_sum_tiles(const xmc_handle* h, int nb, int bpad) {
  if (h->cfg.mode != XMC_MODE_SIMFP8 && 2 * nb <= h->cfg.dim) return 1 << 28;
  const int64_t rows = (int64_t)h->launch_tiles * h->tile_rows / gx_splits(h, h->sm_count, 1, cdiv(h->cfg.dim, 256), bpad);
  return (int)std::max<int64_t>(32, rows / 128);
}

// Whether the one-kernel step is the faster way: with stochastic rounding not for narrow layers at large batches.  What a tile
// costs there for its G and the exchange of its halves grows with the batch, what the kernel saves (fetches of the
// weights) with the features, and of a single box of features one CTA of a cluster does all the rounding.  Three kernels and one, us:
// e4m3 1 000 000 x 64 at batch 40 288 and 288, 72 341 and 391, 128 340 and 392, 500 000 x 128 at 72 199 and 206, 128 199 and 208;
// bf16 1 000 000 x 64 at 64 291 and 309, 128 352 and 354.  A few tiles per cluster are launch latency, and one kernel wins
// everywhere (30 000 x 64 at 128 31.0 and 28.3).  The lines were drawn when the kernel was slower; up to 100 000 rows, and with 192
// features at any batch, it would win beyond them too (100 000 x 128 at 128 57.3 and 54.3, 333 333 x 192 at 128 162 and 142).  Rounded to
// nearest it wins throughout (1 000 000 x 64 at 40 270 and 218, 128 323 and 306, 500 000 x 128 at 128 184 and 166, 333 333 x 192 143 and
// 118) but with the loss beside 64 features (bf16 1 000 000 x 64 at 40 321 and 340).
//
// Simulated FP8, whose three kernels split the embeddings as well, loses by its sums of grad_X having to end (slim_sum_tiles) where a cluster has
// more than 32 tiles, and by the loss, which three kernels add up with sixteen warps.  One kernel and three, us, a cluster's tiles in brackets: 64
// features rounded to nearest [106] at batch 24 185 and 245, 64 253 and 243, 128 283 and 312, with the loss [34] at 16 90 and 95, 64 124 and 97; stochastic
// [11] at 64 44 and 47, [34] 114 and 92, with the loss [11] at 16 43 and 50, 64 52.5 and 51.5; 128 features rounded to nearest [53] at 64 136 and 139, with the
// loss [11] 47 and 51, [22] 81 and 76; stochastic [53] at 24 153 and 158, 64 174 and 156, 96 193 and 193, 128 199 and 199, with the loss [22] at 24 75 and
// 82, [53] 180 and 173, [11] at 64 52 and 56, [22] 92 and 84; 192 with the loss at 64 [16] 72 and 75, [64] 258 and 231, 96 295 and 295; 256 [11] 55 and 66,
// [53] 220 and 216, rounded to nearest 204 and 183; 320 [43] at 96 298 and 318.
bool slim_pays(const xmc_handle* h, int nb, bool sr, bool loss) {
  const int d = h->cfg.dim;
  if (h->cfg.mode == XMC_MODE_SIMFP8) {
    const int tiles = cdiv(slim_tiles(h), h->sm_count / 2);  // of a cluster
    const bool many = tiles > 32;
    if (d > 256 || tiles <= 4) return true;
    if (d > 128) return !(loss && nb == 64 && many);
    if (tiles <= 12) return d == 128 || !(sr && loss) || nb <= 32;
    if (loss) return nb <= 32 && (!sr || (d == 128 && !many));
    if (!sr) return !(d == 64 && nb == 64 && many);
    return d == 128 && nb <= 96 && !(nb == 64 && many);
  }
  return (!sr && (!loss || d > 64)) || 2 * nb <= d || slim_tiles(h) <= 4 * (h->sm_count / 2);
}

}  // namespace

extern "C" {

const char* xmc_last_error(void) { return g_err; }
const char* xmc_version(void) { return "elmo_xmc sm_100a " __DATE__; }

int xmc_create(const xmc_config* cfg, xmc_handle** out) {
  if (cfg == nullptr || out == nullptr) return fail(XMC_ERR_INVALID, "null argument");
  *out = nullptr;
  if (cfg->dim <= 0 || cfg->dim % 64 != 0) return fail(XMC_ERR_INVALID, "dim must be a positive multiple of 64, got %d", cfg->dim);
  if (cfg->max_batch <= 0 || cfg->max_batch > 65535) return fail(XMC_ERR_INVALID, "max_batch must be in [1, 65535], got %d", cfg->max_batch);
  if (cfg->mode < XMC_MODE_BF16 || cfg->mode > XMC_MODE_SIMFP8) return fail(XMC_ERR_INVALID, "unknown mode %d", cfg->mode);
  if (!(cfg->w_scale > 0.f)) return fail(XMC_ERR_INVALID, "w_scale must be positive");
  if (cfg->sched_labels < 0 || cfg->sched_labels % 128 != 0) return fail(XMC_ERR_INVALID, "sched_labels must be a multiple of 128");
  int ndev = 0;
  CU_TRY(cudaGetDeviceCount(&ndev));
  if (cfg->device < 0 || cfg->device >= ndev) return fail(XMC_ERR_INVALID, "device %d out of range (%d devices)", cfg->device, ndev);
  DeviceGuard guard(cfg->device);
  int major = 0, minor = 0, sms = 0, persisting_max = 0;
  CU_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, cfg->device));
  CU_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, cfg->device));
  CU_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, cfg->device));
  CU_TRY(cudaDeviceGetAttribute(&persisting_max, cudaDevAttrMaxPersistingL2CacheSize, cfg->device));
  if (major != 10) return fail(XMC_ERR_CUDA, "device %d is sm_%d%d; this library holds sm_100a code only", cfg->device, major, minor);

  xmc_handle* h = new xmc_handle();
  h->cfg = *cfg;
  h->sm_count = sms;
  h->bpad_max = (int)round_up(cfg->max_batch, 64);
  const int d = cfg->dim;
  // one allocation for what lives as long as the handle
  struct Piece { void** p; size_t bytes; };
  std::vector<Piece> pieces;
  auto A = [&](void** p, size_t bytes) { pieces.push_back({p, (size_t)round_up((long long)bytes, 1024)}); };
  const size_t xrows = (size_t)x_rows_of(h);
  const bool sim = cfg->mode == XMC_MODE_SIMFP8;
  A((void**)&h->x8, (sim ? 4 : 1) * xrows * d);
  A((void**)&h->x16, xrows * d * 2);
  if (sim) {
    A((void**)&h->x_scale, (size_t)round_up((long long)xrows, 256) * 4);       // whole tiles are read
    A((void**)&h->x_wide, (size_t)round_up((long long)xrows, 512));             // so are whole pieces
  }
  A((void**)&h->xt, (size_t)std::max(d, 256) * h->bpad_max * 2);
  // G is sized when the weights are bound
  h->partial_floats = std::max<int64_t>((int64_t)h->sm_count * 256 * 256, (int64_t)h->bpad_max * round_up(d, 256));
  A((void**)&h->partial, (size_t)h->partial_floats * 4);
  A((void**)&h->status, 4 * sizeof(int));
  size_t bytes = 0;
  for (const Piece& piece : pieces) bytes += piece.bytes;
  int rc = dev_alloc(h, &h->arena, bytes, true);
  h->ent_cap = std::max<int64_t>(4096, (int64_t)cfg->max_batch * 64);
  if (rc == XMC_OK) rc = dev_alloc(h, (void**)&h->entries, (size_t)h->ent_cap * 4, false);
  if (rc != XMC_OK) {
    xmc_destroy(h);
    return rc;
  }
  uint8_t* at = reinterpret_cast<uint8_t*>(h->arena);
  for (const Piece& piece : pieces) {
    *piece.p = at;
    at += piece.bytes;
  }
  // L2 carve-out for the partial sums: cudaLimitPersistingL2CacheSize is a limit of the whole CUDA
  // context, so other kernels of the process see that much less L2 while it is set (documented in the
  // header; XMC_NO_L2_PERSIST=1 in the environment leaves the limit alone)
  if (getenv("XMC_NO_L2_PERSIST") == nullptr && persisting_max > 0) {
    const size_t want = std::min<size_t>((size_t)h->partial_floats * 4, (size_t)persisting_max);
    if (cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, want) == cudaSuccess) h->l2_persist_bytes = (int64_t)want;
    else cudaGetLastError();
  }
  *out = h;
  return XMC_OK;
}

int xmc_destroy(xmc_handle* h) {
  if (h == nullptr) return XMC_OK;
  DeviceGuard guard(h->cfg.device);
  if (h->l2_persist_bytes > 0) cudaCtxResetPersistingL2Cache();   // lines pinned for the partial sums become normal again
  void* ptrs[] = {h->w_maps, h->arena, h->G, h->G8, h->xt8, h->bucket_cnt, h->bucket_off, h->entries, h->loss_partial, h->stats, h->topk_gmax, h->topk_run};
  for (void* p : ptrs)
    if (p != nullptr) cudaFree(p);
  for (cudaEvent_t e : h->ev_pool) cudaEventDestroy(e);
  delete h;
  return XMC_OK;
}

int64_t xmc_workspace_bytes(const xmc_handle* h) { return h ? h->ws_bytes : 0; }

int xmc_bind_weights(xmc_handle* h, int32_t n_chunks, void* const* ptrs, const int64_t* rows) {
  if (h == nullptr || ptrs == nullptr || rows == nullptr || n_chunks <= 0) return fail(XMC_ERR_INVALID, "null/empty argument");
  DeviceGuard guard(h->cfg.device);
  int64_t total = 0;
  for (int i = 0; i < n_chunks; ++i) {
    if (ptrs[i] == nullptr || ((uintptr_t)ptrs[i] & 31u)) return fail(XMC_ERR_INVALID, "weight chunk %d: null or not 32-byte aligned", i);
    if (rows[i] <= 0) return fail(XMC_ERR_INVALID, "weight chunk %d has %lld rows", i, (long long)rows[i]);
    if (i + 1 < n_chunks && rows[i] != rows[0]) return fail(XMC_ERR_INVALID, "all weight chunks but the last must have equal rows (chunk %d: %lld vs %lld)", i, (long long)rows[i], (long long)rows[0]);
    if (i + 1 == n_chunks && rows[i] > rows[0]) return fail(XMC_ERR_INVALID, "last weight chunk is larger than the others");
    total += rows[i];
  }
  if (total > (1ll << 31) - 256) return fail(XMC_ERR_INVALID, "too many label rows per handle (%lld)", (long long)total);
  const int d = h->cfg.dim;
  const bool w8 = h->cfg.mode != XMC_MODE_BF16;
  // From here on until everything is there the handle holds no weights: a call after a failure says so.
  {
    std::vector<CUtensorMap> maps((size_t)W_MAPS * n_chunks);
    for (int i = 0; i < n_chunks; ++i) {
      auto at = [&](int kind) { return &maps[(size_t)kind * n_chunks + i]; };
      if (int rc = make_map_kmajor(at(W_ROWS128), w8, ptrs[i], d, rows[i], d, 128)) return rc;
      if (int rc = make_map_kmajor(at(W_ROWS256), w8, ptrs[i], d, rows[i], d, 256)) return rc;
      if (h->cfg.mode == XMC_MODE_SIMFP8) {
        if (int rc = make_map_raw8(at(W_RAW128), ptrs[i], d, rows[i], d, 128)) return rc;
        if (int rc = make_map_raw8(at(W_RAW256), ptrs[i], d, rows[i], d, 256)) return rc;
      }
      // e4m3: raw rows, unswizzled boxes, converted inside the kernel
      if (int rc = make_map_blocked(at(W_GX2), w8, ptrs[i], d, rows[i], d, xmc::kGxRows, !w8, 2)) return rc;
      if (int rc = make_map_blocked(at(W_GX4), w8, ptrs[i], d, rows[i], d, xmc::kGxRows, !w8, 4)) return rc;
    }
    h->w_ptrs.clear();
    if (h->w_maps) { cudaFree(h->w_maps); h->ws_bytes -= h->w_maps_bytes; h->w_maps = nullptr; }
    h->w_maps_bytes = (int64_t)(maps.size() * sizeof(CUtensorMap));
    if (int rc = dev_alloc(h, (void**)&h->w_maps, (size_t)h->w_maps_bytes, false)) return rc;
    CU_TRY(cudaMemcpy(h->w_maps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice));
    if (int rc = host_work_done()) return rc;
  }
  h->w_rows.assign(rows, rows + n_chunks);
  h->total_rows = total;
  h->rows_per_chunk = rows[0];
  int max_pairs = 0;
  if (int rc = gradx_configure(h->sm_count, &max_pairs)) return rc;
  const bool pairs = use_pairs(max_pairs);
  const int workers = pairs ? max_pairs : h->sm_count;
  h->tile_rows = pairs ? 256 : 128;
  h->tiles_per_chunk = cdiv(rows[0], h->tile_rows);
  h->n_tiles = (n_chunks - 1) * h->tiles_per_chunk + cdiv(rows[n_chunks - 1], h->tile_rows);
  // Label tiles per launch: long launches, because each one pays the kernels' ramps and half-empty last rounds once;
  // bounded by the memory of their G: 64 MB, more for large weights (an eighth of them) and large batches (a
  // launch of 65 536 rows), up to 128 MB, and a quarter on top.  The launches are made equal and, where that
  // fits, a multiple of the CTA pairs the device holds, so that a last round of tiles is full.
  // 670 091 x 768 e4m3, batch 256: 5 launches of each kernel instead of 11, step 960 -> 860 us.  (131 072 rows and 256 MB would take 2 % off
  // 2 812 281 x 768 at batch 1024, but a sum of grad_X is as long as a launch over its splits, and over e4m3 weights nothing else ends it.)
  const int64_t tile_bytes = (int64_t)h->tile_rows * h->bpad_max * 2;
  if (h->cfg.sched_labels > 0) {
    h->launch_tiles = (int)std::max<int64_t>(1, h->cfg.sched_labels / h->tile_rows);
  } else {
    const int64_t by_weights = total * d * (w8 ? 1 : 2) / 8, by_batch = std::min<int64_t>(65536, rows[0]) * h->bpad_max * 2;
    const int64_t budget = std::max<int64_t>(64ll << 20, std::min<int64_t>(128ll << 20, std::max(by_weights, by_batch)));
    const int64_t most = std::max<int64_t>(1, budget * 5 / 4 / tile_bytes);
    const int64_t per = cdiv(h->n_tiles, cdiv(h->n_tiles, most)), up = round_up(per, workers);
    h->launch_tiles = (int)(per > workers && up <= most ? up : per);
  }
  h->launch_tiles = std::min(h->launch_tiles, h->n_tiles);
  const int64_t g_rows = (int64_t)h->launch_tiles * h->tile_rows;
  if (g_rows > h->g_rows) {
    // whole multiples of 256 rows: the fused top-k keeps windows of logits in here
    if (h->G) { cudaFree(h->G); h->ws_bytes -= round_up(h->g_rows, 256) * h->bpad_max * 2; h->G = nullptr; }
    if (h->G8) { cudaFree(h->G8); h->ws_bytes -= h->g8_rows * h->bpad_max; h->G8 = nullptr; h->g8_rows = 0; }
    h->g_rows = 0;
    if (int rc = dev_alloc(h, (void**)&h->G, (size_t)round_up(g_rows, 256) * h->bpad_max * 2, true)) return rc;
    h->g_rows = g_rows;
  }
  const int nb = n_chunks * cdiv(rows[0], 128);
  const int64_t loss_cap = (int64_t)cdiv(h->n_tiles, h->launch_tiles) * h->sm_count * xmc::kMaxEpiWarps;
  if (nb != h->n_buckets || loss_cap != h->loss_cap) {
    if (h->bucket_cnt) { cudaFree(h->bucket_cnt); h->ws_bytes -= (int64_t)h->n_buckets * 8; h->bucket_cnt = nullptr; }
    if (h->bucket_off) { cudaFree(h->bucket_off); h->ws_bytes -= (int64_t)(h->n_buckets + 1) * 4; h->bucket_off = nullptr; }
    if (h->loss_partial) { cudaFree(h->loss_partial); h->ws_bytes -= h->loss_cap * 8; h->loss_partial = nullptr; }
    h->n_buckets = nb;
    h->loss_cap = loss_cap;
    int rc = dev_alloc(h, (void**)&h->bucket_cnt, (size_t)nb * 8, true);
    if (rc == XMC_OK) rc = dev_alloc(h, (void**)&h->bucket_off, (size_t)(nb + 1) * 4, true);
    if (rc == XMC_OK) rc = dev_alloc(h, (void**)&h->loss_partial, (size_t)h->loss_cap * 8, true);
    if (rc != XMC_OK) {
      h->loss_cap = -1;                    // not what any binding asks for: the next one starts here again
      return rc;
    }
  }
  h->w_ptrs.assign(ptrs, ptrs + n_chunks);
  return XMC_OK;
}

int xmc_bind_kahan(xmc_handle* h, void* buf, int64_t rows, int32_t dtype) {
  if (h == nullptr) return fail(XMC_ERR_INVALID, "null handle");
  if (buf == nullptr || rows == 0) {
    h->kahan = nullptr;
    h->kahan_rows = 0;
    return XMC_OK;
  }
  if (h->cfg.mode != XMC_MODE_FP8) return fail(XMC_ERR_STATE, "the Kahan head is defined for the real-FP8 mode only");
  if (h->w_ptrs.empty()) return fail(XMC_ERR_STATE, "bind the weights first");
  if (dtype != XMC_DT_BF16 && dtype != XMC_DT_E5M2) return fail(XMC_ERR_INVALID, "compensation buffer must be bf16 or e5m2");
  if (rows < 0 || rows > h->w_rows[0]) return fail(XMC_ERR_INVALID, "head rows %lld exceed the first weight chunk (%lld rows)", (long long)rows, (long long)h->w_rows[0]);
  if ((uintptr_t)buf & 15u) return fail(XMC_ERR_INVALID, "compensation buffer not 16-byte aligned");
  h->kahan = buf;
  h->kahan_rows = rows;
  h->kahan_e5m2 = dtype == XMC_DT_E5M2 ? 1 : 0;
  return XMC_OK;
}

int xmc_weight_stats(xmc_handle* h, int64_t* counts, float* amax_stored, void* stream) {
  if (h == nullptr || counts == nullptr || amax_stored == nullptr) return fail(XMC_ERR_INVALID, "null argument");
  if (h->w_ptrs.empty()) return fail(XMC_ERR_STATE, "xmc_bind_weights has not been called");
  if (h->cfg.mode == XMC_MODE_BF16) return fail(XMC_ERR_STATE, "weight statistics are defined for e4m3 weights");
  DeviceGuard guard(h->cfg.device);
  cudaStream_t st = (cudaStream_t)stream;
  if (h->stats == nullptr) {
    if (int rc = dev_alloc(h, (void**)&h->stats, 8 * sizeof(unsigned long long), true)) return rc;
  }
  CU_TRY(cudaMemsetAsync(h->stats, 0, 8 * sizeof(unsigned long long), st));
  const int d = h->cfg.dim;
  for (size_t wc = 0; wc < h->w_ptrs.size(); ++wc) {
    const long long n16 = (long long)h->w_rows[wc] * d / 16;
    const int blocks = (int)std::min<long long>((n16 + 255) / 256, (long long)h->sm_count * 8);
    xmc::weight_stats_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<const uint4*>(h->w_ptrs[wc]), n16, h->stats,
                                                     reinterpret_cast<unsigned int*>(h->stats + 4));
    CU_TRY(cudaGetLastError());
  }
  unsigned long long host[8];
  CU_TRY(cudaMemcpyAsync(host, h->stats, sizeof(host), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  for (int i = 0; i < 4; ++i) counts[i] = (int64_t)host[i];
  counts[4] = h->total_rows * d;
  // magnitude byte -> value: exponent field e, mantissa m: e ? 2^(e-7) (1 + m/8) : m 2^-9
  const unsigned int mb = (unsigned int)(host[4] & 0x7Fu);
  const int e = (int)(mb >> 3), m = (int)(mb & 7u);
  *amax_stored = e ? ldexpf(1.0f + (float)m / 8.0f, e - 7) : ldexpf((float)m, -9);
  return XMC_OK;
}

int xmc_rescale(xmc_handle* h, int32_t shift, int32_t stochastic, uint64_t seed, uint64_t step, void* stream) {
  if (h == nullptr) return fail(XMC_ERR_INVALID, "null handle");
  if (h->w_ptrs.empty()) return fail(XMC_ERR_STATE, "xmc_bind_weights has not been called");
  if (h->cfg.mode == XMC_MODE_BF16) return fail(XMC_ERR_STATE, "the per-tensor scale belongs to e4m3 weights");
  if (shift < -16 || shift > 16) return fail(XMC_ERR_INVALID, "shift %d outside [-16, 16]", shift);
  if (h->kahan != nullptr && shift != 0) return fail(XMC_ERR_STATE, "rescaling with a Kahan head bound is not defined");
  if (shift == 0) return XMC_OK;
  DeviceGuard guard(h->cfg.device);
  cudaStream_t st = (cudaStream_t)stream;
  const int d = h->cfg.dim;
  const float factor = ldexpf(1.0f, -shift);
  int64_t row_base = 0;
  for (size_t wc = 0; wc < h->w_ptrs.size(); ++wc) {
    const long long n8 = (long long)h->w_rows[wc] * d / 8;
    const int blocks = (int)std::min<long long>((n8 + 255) / 256, (long long)h->sm_count * 8);
    xmc::rescale_e4m3_kernel<<<blocks, 256, 0, st>>>(reinterpret_cast<uint2*>(h->w_ptrs[wc]), n8, factor, stochastic ? 1 : 0,
                                                     seed, step, (unsigned long long)(h->cfg.label_offset + row_base) * d);
    CU_TRY(cudaGetLastError());
    row_base += h->w_rows[wc];
  }
  h->cfg.w_scale = ldexpf(h->cfg.w_scale, shift);
  return XMC_OK;
}

float xmc_get_scale(const xmc_handle* h) { return h ? h->cfg.w_scale : 0.f; }

int xmc_set_scale(xmc_handle* h, float scale) {
  if (h == nullptr) return fail(XMC_ERR_INVALID, "null handle");
  if (!(scale > 0.f)) return fail(XMC_ERR_INVALID, "w_scale must be positive");
  h->cfg.w_scale = scale;
  return XMC_OK;
}

int xmc_check(xmc_handle* h, void* stream) {
  if (h == nullptr) return fail(XMC_ERR_INVALID, "null handle");
  DeviceGuard guard(h->cfg.device);
  cudaStream_t st = (cudaStream_t)stream;
  CU_TRY(cudaStreamSynchronize(st));
  int host[4] = {0, 0, 0, 0};
  CU_TRY(cudaMemcpy(host, h->status, sizeof(host), cudaMemcpyDeviceToHost));
  if (host[0] != xmc::DEV_OK) {
    CU_TRY(cudaMemset(h->status, 0, sizeof(host)));
    if (host[0] == xmc::DEV_WAIT_TIMEOUT)
      return fail(XMC_ERR_DEVICE_FLAG, "kernel wait timed out (block %d, site %d)", host[1], host[2]);
    if (host[0] == xmc::DEV_BAD_LABEL)
      return fail(XMC_ERR_DEVICE_FLAG, "label pair with batch row out of range or negative id (row %d)", host[2]);
    return fail(XMC_ERR_DEVICE_FLAG, "device status %d (block %d, info %d)", host[0], host[1], host[2]);
  }
  return XMC_OK;
}

int xmc_step(xmc_handle* h, const void* x, int32_t x_dtype, int32_t batch, const int32_t* labels,
             int64_t nnz, float lr, float wd, uint64_t seed, uint64_t step, uint32_t flags,
             float* grad_x_f32, void* grad_x_bf16, double* loss_out, void* stream) {
  if (h == nullptr || x == nullptr) return fail(XMC_ERR_INVALID, "null argument");
  if (h->w_ptrs.empty()) return fail(XMC_ERR_STATE, "xmc_bind_weights has not been called");
  if (x_dtype != XMC_DT_BF16) return fail(XMC_ERR_INVALID, "xmc_step takes bf16 embeddings");
  if (batch <= 0 || batch > h->cfg.max_batch) return fail(XMC_ERR_INVALID, "batch %d outside [1, %d]", batch, h->cfg.max_batch);
  if (nnz < 0 || (nnz > 0 && labels == nullptr)) return fail(XMC_ERR_INVALID, "labels missing");
  if ((flags & XMC_STEP_COMPUTE_LOSS) && loss_out == nullptr) return fail(XMC_ERR_INVALID, "loss_out missing");
  if (((uintptr_t)grad_x_f32 & 15u) || ((uintptr_t)grad_x_bf16 & 1u)) return fail(XMC_ERR_INVALID, "grad_x not aligned");
  DeviceGuard guard(h->cfg.device);
  cudaStream_t st = (cudaStream_t)stream;
  const int d = h->cfg.dim, mode = h->cfg.mode;
  const int bpad = (int)round_up(batch, 64);   // G rows are fetched in blocks of 64 batch columns
  const bool w8 = mode != XMC_MODE_BF16;
  const bool fwd_fp8 = mode == XMC_MODE_FP8, sim = mode == XMC_MODE_SIMFP8;
  const bool want_loss = (flags & XMC_STEP_COMPUTE_LOSS) != 0;
  const bool sr = (flags & XMC_STEP_STOCHASTIC) != 0;
  const bool dw8 = (flags & XMC_STEP_FP8_DW) != 0;
  if (dw8) {
    if (!fwd_fp8) return fail(XMC_ERR_STATE, "the FP8 dW contraction belongs to the real-FP8 mode");
    if ((flags & XMC_STEP_ROUND_DW_BF16) || wd != 0.f || h->kahan != nullptr)
      return fail(XMC_ERR_STATE, "the FP8 dW contraction takes no weight decay, bf16 dW rounding or Kahan head");
    if (h->G8 == nullptr || h->g8_rows < h->g_rows) {
      CU_TRY(cudaStreamSynchronize(st));
      if (h->G8) { cudaFree(h->G8); h->ws_bytes -= h->g8_rows * h->bpad_max; h->G8 = nullptr; }
      if (int rc = dev_alloc(h, (void**)&h->G8, (size_t)h->g_rows * h->bpad_max, true)) return rc;
      h->g8_rows = h->g_rows;
    }
    if (h->xt8 == nullptr) {
      if (int rc = dev_alloc(h, (void**)&h->xt8, (size_t)std::max(h->cfg.dim, 256) * h->bpad_max, true)) return rc;
    }
  }

  int gx_max_pairs = 0;
  if (int rc = gradx_configure(h->sm_count, &gx_max_pairs)) return rc;
  const bool pairs_ok = use_pairs(gx_max_pairs);          // a device that cannot hold a pair runs everything on single CTAs
  xmc::SlimParams sp;
  int slim_smem = 0;
  // (dW as the two reference layers have it: in bf16 with bf16 weights, not rounded with e4m3 ones)
  const bool slim = pairs_ok && !dw8 && wd == 0.f && ((flags & XMC_STEP_ROUND_DW_BF16) != 0) == !w8 &&
                    slim_geometry(w8, sim, h->kahan != nullptr, want_loss, batch, d, &sp, &slim_smem) && slim_pays(h, sp.nb, sr, want_loss);

  // --- embeddings: e4m3 copy (forward), bf16 copy, bf16 transpose (update); positives bucketed by label tile ---
  if (nnz > h->ent_cap) {
    CU_TRY(cudaStreamSynchronize(st));
    CU_TRY(cudaFree(h->entries));
    h->ws_bytes -= h->ent_cap * 4;
    h->entries = nullptr;
    h->ent_cap = 0;
    const int64_t want = nnz + nnz / 2;
    if (int rc = dev_alloc(h, (void**)&h->entries, (size_t)want * 4, false)) return rc;
    h->ent_cap = want;
  }
  const xmc::BucketGeom geom = geom_of(h);
  const size_t bucket_smem = (size_t)(h->n_buckets + 1) * 4;
  // One block can sort a few thousand pairs while the others prepare X, if the counts fit into the shared memory a
  // kernel gets without asking (40 KB: 1.3 M labels) and the pairs are read as 8-byte words; a block sorts about 700
  // pairs a microsecond, four more launches cost about 10 (12 543 pairs: step of 100 000 x 256, batch 512 168 us by one block, 160).
  // Up to a thousand pairs are sorted by blocks of 256 threads, which start and meet faster (step of 31 003 x 768, batch 16
  // with 80 pairs, 256 and 1024 threads: 41.4 and 41.9 us), more by 1024 (31 003 x 256, batch 256 with 5 000: 54.1 and 51.4);
  // beyond batch 128 X is what takes the time (31 003 x 768 at 140 with 140 pairs 57.0 and 55.5).
  if (nnz <= 8192 && bucket_smem <= 40960 && ((uintptr_t)labels & 7u) == 0) {
    const bool few = nnz <= 1024 && batch <= 128;
    int x_blocks;
    const xmc::PrepX px = prep_args(h, x, x_dtype, batch, bpad, fwd_fp8, !w8, !dw8, dw8, sim, &x_blocks);
    mark(h, K_PREP, st);
    const auto kernel = px.row_blocks > 0 ? few ? xmc::prep_step_kernel<256, 4, true> : batch <= 128 ? xmc::prep_step_kernel<1024, 8, true> : xmc::prep_step_kernel<1024, 0, true>
                                          : few ? xmc::prep_step_kernel<256, 4, false> : batch <= 128 ? xmc::prep_step_kernel<1024, 8, false> : xmc::prep_step_kernel<1024, 0, false>;
    CU_TRY(launch_pdl(kernel, 1 + x_blocks, few ? 256 : 1024,
                      bucket_smem, st, px, labels, (int)nnz, geom, h->bucket_off, h->entries, h->status, slim ? 1 : 0));
  } else {
    if (int rc = prep_x(h, x, x_dtype, batch, bpad, fwd_fp8, !w8, !dw8, st, dw8, sim)) return rc;
    CU_TRY(cudaMemsetAsync(h->bucket_cnt, 0, (size_t)h->n_buckets * 8, st));
    const int blocks = std::max(1, cdiv(nnz, 256));
    mark(h, K_PREP, st);
    CU_TRY(launch_pdl(xmc::bucket_count_kernel, blocks, 256, 0, st, labels, (long long)nnz, (int)batch, geom, h->bucket_cnt, h->status));
    mark(h, K_PREP, st);
    CU_TRY(launch_pdl(xmc::bucket_scan_kernel, 1, 1024, 0, st, (const int*)h->bucket_cnt, h->n_buckets, h->bucket_off));
    mark(h, K_PREP, st);
    CU_TRY(launch_pdl(xmc::bucket_fill_kernel, blocks, 256, 0, st, labels, (long long)nnz, (int)batch, geom, (const int*)h->bucket_off,
                      h->bucket_cnt + h->n_buckets, h->entries));
  }

  const float lr_eff = lr / h->cfg.w_scale;
  size_t loss_slots = 0;
  auto reduce = [&](int n_splits, int slot_rows) -> int {
    const bool grad = grad_x_f32 != nullptr || grad_x_bf16 != nullptr;
    if (grad || want_loss) {
      const int blocks = (grad ? std::min(cdiv((long long)batch * d, 128), h->sm_count * 8) : 0) + (want_loss ? 1 : 0);
      const xmc::LossSum loss = {h->loss_partial, want_loss ? (int)loss_slots : 0, loss_out};
      mark(h, K_REDUCE, st);
      CU_TRY(launch_pdl(xmc::reduce_gradx_kernel, blocks, xmc::kReduceThreads, 0, st, (const float*)h->partial, n_splits, (int)batch,
                        slot_rows, d, h->cfg.w_scale, grad_x_f32, reinterpret_cast<__nv_bfloat16*>(grad_x_bf16), loss));
    }
    return XMC_OK;
  };

  // --- small batches: the whole step in one kernel ---
  if (slim) {
    CUtensorMap map_x, map_xt;
    const size_t xrows = (size_t)x_rows_of(h);
    if (int rc = sim ? make_map_parts(h, &map_x, sp.nb / 2)
                     : make_map_kmajor(&map_x, w8, w8 ? (const void*)h->x8 : (const void*)h->x16, d, xrows, d, (uint32_t)sp.nb / 2)) return rc;
    if (int rc = make_map_kmajor(&map_xt, false, h->xt, bpad, std::max(d, 256), bpad, (uint32_t)sp.uw)) return rc;
    const int tpc = cdiv(h->rows_per_chunk, 128);
    sp.w_maps = chunk_maps(h, W_ROWS128);
    sp.n_chunks = (int)h->w_ptrs.size();
    sp.rows_full = (int)h->rows_per_chunk;
    sp.rows_last = (int)h->w_rows.back();
    sp.n_tiles = slim_tiles(h);
    sp.div_tpc = xmc::make_fastdiv(tpc, sp.n_tiles);
    sp.bkt_per_chunk = geom.per_chunk;
    sp.batch = batch;
    sp.gx_mask = kSlimChainTiles - 1;
    sp.gx_tiles = slim_sum_tiles(h, sp.nb, bpad);
    sp.w_scale = h->cfg.w_scale;
    sp.x_scale = h->x_scale;
    sp.part_rows = x_rows_of(h);
    sp.x_wide = h->x_wide;
    sp.bucket_off = h->bucket_off;
    sp.bucket_ent = h->entries;
    sp.loss_partial = want_loss ? h->loss_partial : nullptr;
    sp.partial = h->partial;
    sp.status = h->status;
    memset(&sp.upd, 0, sizeof(sp.upd));
    fill_update_stream(&sp.upd, seed, step, lr_eff, 0.f);
    sp.upd.d = d;
    sp.upd.elem0 = (unsigned long long)h->cfg.label_offset * (unsigned long long)d;
    sp.upd.kahan = h->kahan;
    sp.upd.kahan_rows = (int)h->kahan_rows;
    sp.upd.kahan_e5m2 = h->kahan_e5m2;
    const int max_clusters = (int)std::min<int64_t>(h->sm_count / 2, h->partial_floats / ((int64_t)sp.nb * d));
    int grid = 0, rc;
    mark(h, K_UPD, st);
    auto as = [&](auto launch) { return launch(map_x, map_xt, sp, slim_smem, max_clusters, h->sm_count, st, &grid); };
    auto of_terms = [&](auto sr_, auto loss_, auto terms_) -> int {
      constexpr bool SR = decltype(sr_)::value, LOSS = decltype(loss_)::value;
      constexpr xmc::KahanTerms TERMS = decltype(terms_)::value;
      constexpr bool BOUND = !SR && TERMS == xmc::kKahanNone;
      return sp.nb > 64 ? as(launch_slim<true, SR, LOSS, TERMS, false, false, BOUND>) : as(launch_slim<true, SR, LOSS, TERMS, true, false, BOUND>);
    };
    auto of_weights = [&](auto sr_, auto loss_) -> int {
      if (!w8) {
        constexpr bool SR = decltype(sr_)::value, LOSS = decltype(loss_)::value;
        return sp.nb > 64 ? as(launch_slim<false, SR, LOSS, xmc::kKahanNone, false>) : as(launch_slim<false, SR, LOSS, xmc::kKahanNone, true>);
      }
      if (sim) {
        constexpr bool SR = decltype(sr_)::value, LOSS = decltype(loss_)::value;
        if (cdiv(sp.n_tiles, std::min(max_clusters, gx_max_pairs)) > sp.gx_tiles)
          return sp.nb > 64 ? as(launch_slim<true, SR, LOSS, xmc::kKahanNone, false, true, true>) : as(launch_slim<true, SR, LOSS, xmc::kKahanNone, true, true, true>);
        return sp.nb > 64 ? as(launch_slim<true, SR, LOSS, xmc::kKahanNone, false, true>) : as(launch_slim<true, SR, LOSS, xmc::kKahanNone, true, true>);
      }
      if (h->kahan == nullptr) return of_terms(sr_, loss_, std::integral_constant<xmc::KahanTerms, xmc::kKahanNone>());
      if (h->kahan_e5m2) return of_terms(sr_, loss_, std::integral_constant<xmc::KahanTerms, xmc::kKahanE5m2>());
      return of_terms(sr_, loss_, std::integral_constant<xmc::KahanTerms, xmc::kKahanBf16>());
    };
    const std::true_type yes;
    const std::false_type no;
    if (sr) rc = want_loss ? of_weights(yes, yes) : of_weights(yes, no);
    else rc = want_loss ? of_weights(no, yes) : of_weights(no, no);
    if (rc) return rc;
    loss_slots = (size_t)grid * xmc::kSlGWarps;
    if (int rc2 = reduce(grid / 2, sp.nb)) return rc2;
    mark(h, K_END, st);
    return XMC_OK;
  }

  // --- grad_X partial geometry ---
  // On CTA pairs where every feature tile is whole and both CTAs of a pair have batch rows to work on; otherwise one CTA per
  // 256 x 256 tile.  A pair takes 512 batch rows of e4m3 weights, which it has to convert, else 256.  (e4m3 weights at
  // batches up to 192 would be faster on pairs too, 52.5 -> 47.3 us for 131 072 x 768, but with half as many splits their
  // unbounded sums are twice as long.  Weights U(+-1/sqrt(d)) do not show that, 670 091 x 768 at 140 4.9e-8 and 5.0e-8; spread
  // evenly over ten binades they do, 2.1e-6 and 4.9e-6, all of one sign 2.3e-6 and 8.4e-6.)
  const int n_dt = cdiv(d, 256);
  const bool pair_gx = pairs_ok && d % 256 == 0 && bpad >= (w8 ? 256 : 192);
  const int gx_halves = pair_gx && (!w8 || bpad <= 256) ? 1 : 2;
  const int n_bt = cdiv(bpad, pair_gx ? gx_halves * 256 : 256);
  const int n_splits = gx_splits(h, pair_gx ? gx_max_pairs : h->sm_count, n_bt, n_dt, bpad);
  if ((int64_t)n_splits * bpad * d > h->partial_floats) return fail(XMC_ERR_STATE, "grad_X workspace too small");

  // Keep the grad_X partial sums resident in L2 across the chunk launches of this step: every
  // grad_X launch re-reads and re-writes them, and the weights/G streaming through L2 in between
  // would otherwise push them out to HBM each time.  The window covers only this private buffer.
  if (h->l2_persist_bytes > 0) {
    cudaStreamAttrValue attr;
    memset(&attr, 0, sizeof(attr));
    attr.accessPolicyWindow.base_ptr = h->partial;
    attr.accessPolicyWindow.num_bytes = std::min<size_t>((size_t)n_splits * bpad * d * 4, (size_t)h->l2_persist_bytes);
    attr.accessPolicyWindow.hitRatio = 1.0f;
    attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
    attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    CU_TRY(cudaStreamSetAttribute(st, cudaStreamAttributeAccessPolicyWindow, &attr));
  }

  // --- operand maps that do not change across chunks ---
  CUtensorMap map_x, map_xt, map_g_k, map_g_mn;
  const size_t xrows = (size_t)x_rows_of(h);
  // CTA pairs (256-row label tiles, each CTA staging half of the other operand's rows) for the kernels
  // of the forward and the update
  const uint32_t half = pairs_ok ? 128 : 256;
  // a single batch tile: boxes of X hold the columns that its MMAs read
  const uint32_t x_rows = bpad < 256 ? (uint32_t)(pairs_ok ? bpad / 2 : bpad) : half;
  if (int rc = sim ? make_map_parts(h, &map_x, (int)x_rows)
                   : make_map_kmajor(&map_x, w8, w8 ? (const void*)h->x8 : (const void*)h->x16, d, xrows, d, x_rows)) return rc;
  if (dw8) {
    if (int rc = make_map_kmajor(&map_xt, true, h->xt8, bpad, std::max(d, 256), bpad, half)) return rc;
    if (int rc = make_map_kmajor(&map_g_k, true, h->G8, bpad, h->g8_rows, bpad, 128)) return rc;
  } else {
    if (int rc = make_map_kmajor(&map_xt, false, h->xt, bpad, std::max(d, 256), bpad, half)) return rc;
    if (int rc = make_map_kmajor(&map_g_k, false, h->G, bpad, h->g_rows, bpad, 128)) return rc;
  }
  if (int rc = make_map_blocked(&map_g_mn, false, h->G, bpad, h->g_rows, bpad, xmc::kGxRows, true, pair_gx ? 2 : 4)) return rc;

  // G as the forward stores it: boxes of 32 label rows x 64 batch columns
  CUtensorMap map_g_out;
  if (int rc = make_map(&map_g_out, false, h->G, bpad, h->g_rows, (uint64_t)bpad * 2, 64, 32)) return rc;

  for (int t0 = 0; t0 < h->n_tiles; t0 += h->launch_tiles) {
    const int n_lt = std::min(h->launch_tiles, h->n_tiles - t0);
    const xmc::LabelTiles lt = label_tiles(h, h->tile_rows, t0, n_lt);

    // forward + loss gradient -> G
    xmc::FwdParams fp;
    fp.after_prep = t0 == 0 ? 1 : 0;
    fp.lt = lt;
    fp.w_maps = chunk_maps(h, W_ROWS128);
    fp.n_btiles = cdiv(bpad, 256);
    const int f_tiles = n_lt * fp.n_btiles;
    fp.div_btiles = xmc::make_fastdiv(fp.n_btiles, f_tiles);
    fp.batch = batch;
    fp.bpad = bpad;
    fp.x_rows = (int)x_rows;
    fp.k_steps = cdiv((long long)d * (w8 ? 1 : 2), 128);
    fp.w_scale = h->cfg.w_scale;
    fp.x_scale = h->x_scale;
    fp.part_rows = x_rows_of(h);
    fp.x_wide = h->x_wide;
    fp.G = h->G;
    fp.G8 = h->G8;
    fp.bucket_off = h->bucket_off;
    fp.bucket_ent = h->entries;
    fp.bkt_per_chunk = geom.per_chunk;
    fp.loss_partial = want_loss ? h->loss_partial + loss_slots : nullptr;
    fp.status = h->status;
    int rc, f_grid = 0;
    mark(h, K_FWD, st);
#define XMC_FWD(PAIR_, FP8_, G8_, SPLIT_) \
  (want_loss ? launch_gemm<xmc::FwdPolicy<FP8_, true, G8_, SPLIT_>, PAIR_>(map_x, map_x, fp, f_tiles, h->sm_count, st, 0, &map_g_out, &f_grid) \
             : launch_gemm<xmc::FwdPolicy<FP8_, false, G8_, SPLIT_>, PAIR_>(map_x, map_x, fp, f_tiles, h->sm_count, st, 0, &map_g_out, &f_grid))
    if (sim) rc = pairs_ok ? XMC_FWD(true, true, false, true) : XMC_FWD(false, true, false, true);
    else if (dw8) rc = pairs_ok ? XMC_FWD(true, true, true, false) : XMC_FWD(false, true, true, false);
    else if (fwd_fp8) rc = pairs_ok ? XMC_FWD(true, true, false, false) : XMC_FWD(false, true, false, false);
    else rc = pairs_ok ? XMC_FWD(true, false, false, false) : XMC_FWD(false, false, false, false);
#undef XMC_FWD
    if (rc) return rc;
    // every epilogue warp of every launched CTA writes its slot: launches append, nothing has to be cleared
    if (want_loss) loss_slots += (size_t)f_grid * xmc::kMaxEpiWarps;

    // grad_X partials: uses the pre-update weights (reference: chunked.py:116 precedes :119-127)
    const int ksteps_per_tile = h->tile_rows / xmc::kGxRows;
    xmc::GxParams gp;
    gp.bpad = bpad;
    gp.d = d;
    gp.n_btiles = n_bt;
    gp.n_dtiles = n_dt;
    gp.n_splits = n_splits;
    gp.total_ksteps = n_lt * ksteps_per_tile;
    gp.w_maps = chunk_maps(h, pair_gx ? W_GX2 : W_GX4);
    gp.first_kstep = t0 * ksteps_per_tile;
    gp.ksteps_per_chunk = h->tiles_per_chunk * ksteps_per_tile;
    gp.accumulate = t0 == 0 ? 0 : 1;
    // (on pairs the end of a segment costs next to nothing)
    gp.chain_ksteps = cdiv(pair_gx ? kMinChainRows : std::max(kMinChainRows, cdiv(kChainRows, n_splits)), xmc::kGxRows);
    gp.partial = h->partial;
    gp.status = h->status;
    mark(h, K_GRADX, st);
    {
      const int grid = n_bt * n_dt * n_splits;
      if (pair_gx) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[2];
        const int smem = !w8 ? xmc::kGxSmemBytes<false, true, 1> : gx_halves == 1 ? xmc::kGxSmemBytes<true, true, 1> : xmc::kGxSmemBytes<true, true, 2>;
        launch_config(&cfg, at, 2 * grid, xmc::kGxThreads, smem, st, 2);
        CU_TRY(cudaLaunchKernelEx(&cfg, !w8 ? xmc::gradx_kernel<false, true, 1> : gx_halves == 1 ? xmc::gradx_kernel<true, true, 1> : xmc::gradx_kernel<true, true, 2>,
                                  map_g_mn, map_g_mn, gp));
      } else if (w8) {
        CU_TRY(launch_pdl(xmc::gradx_kernel<true>, grid, xmc::kGxThreads, xmc::kGxSmemBytes<true, false, 2>, st, map_g_mn, map_g_mn, gp));
      } else {
        CU_TRY(launch_pdl(xmc::gradx_kernel<false>, grid, xmc::kGxThreads, xmc::kGxSmemBytes<false, false, 2>, st, map_g_mn, map_g_mn, gp));
      }
    }

    // fused dW + SGD update of the tiles' weights, in place
    xmc::UpdParams up;
    up.lt = lt;
    up.w_maps = chunk_maps(h, W_ROWS128);
    up.n_dtiles = n_dt;
    const int u_tiles = n_lt * n_dt;
    up.div_dtiles = xmc::make_fastdiv(n_dt, u_tiles);
    up.d = d;
    up.k_steps = cdiv(bpad, dw8 ? 128 : 64);
    fill_update_stream(&up, seed, step, dw8 ? lr_eff / xmc::kG8Scale : lr_eff, wd);
    up.elem0 = (unsigned long long)h->cfg.label_offset * (unsigned long long)d;
    up.round_dw_bf16 = (flags & XMC_STEP_ROUND_DW_BF16) ? 1 : 0;
    up.status = h->status;
    mark(h, K_UPD, st);
    // the reference pairs: e4m3 weights (no dW rounding), bf16 weights (dW materialised in bf16);
    // weight decay is off in both, so only those combinations get the branch-free fast kernels
    up.kahan = h->kahan;
    up.kahan_rows = (int)h->kahan_rows;
    up.kahan_e5m2 = h->kahan_e5m2;
    const bool kahan_here = h->kahan != nullptr && (int64_t)t0 * h->tile_rows < h->kahan_rows;
    const bool rdw = up.round_dw_bf16 != 0, has_wd = wd != 0.f;
    if (kahan_here && (!w8 || rdw || has_wd)) return fail(XMC_ERR_STATE, "the Kahan head needs e4m3 weights without weight decay");
#define XMC_UPD(...) \
  (pairs_ok ? launch_gemm<xmc::UpdPolicy<__VA_ARGS__>, true>(map_g_k, map_xt, up, u_tiles, h->sm_count, st) \
            : launch_gemm<xmc::UpdPolicy<__VA_ARGS__>, false>(map_g_k, map_xt, up, u_tiles, h->sm_count, st))
    if (dw8) {
      rc = sr ? XMC_UPD(true, true, false, false, false, true) : XMC_UPD(true, false, false, false, false, true);
    } else if (kahan_here) {
      rc = sr ? XMC_UPD(true, true, false, false, true) : XMC_UPD(true, false, false, false, true);
    } else if (w8) {
      if (!rdw && !has_wd) rc = sr ? XMC_UPD(true, true, false, false) : XMC_UPD(true, false, false, false);
      else if (!rdw) rc = sr ? XMC_UPD(true, true, false, true) : XMC_UPD(true, false, false, true);
      else rc = sr ? XMC_UPD(true, true, true, true) : XMC_UPD(true, false, true, true);
    } else {
      if (rdw && !has_wd) rc = sr ? XMC_UPD(false, true, true, false) : XMC_UPD(false, false, true, false);
      else if (rdw) rc = sr ? XMC_UPD(false, true, true, true) : XMC_UPD(false, false, true, true);
      else rc = sr ? XMC_UPD(false, true, false, true) : XMC_UPD(false, false, false, true);
    }
#undef XMC_UPD
    if (rc) return rc;
  }

  if (int rc = reduce(n_splits, bpad)) return rc;
  if (h->l2_persist_bytes > 0) {
    // the caller's stream leaves this call without the window (kernels launched after it are unaffected)
    cudaStreamAttrValue attr;
    memset(&attr, 0, sizeof(attr));
    CU_TRY(cudaStreamSetAttribute(st, cudaStreamAttributeAccessPolicyWindow, &attr));
  }
  mark(h, K_END, st);
  return XMC_OK;
}

int64_t xmc_launch_count(const xmc_handle* h) { return h ? h->launches : 0; }

int xmc_profile(xmc_handle* h, int32_t enable, double* ms_by_kind, int64_t* launches_by_kind) {
  if (h == nullptr) return fail(XMC_ERR_INVALID, "null handle");
  DeviceGuard guard(h->cfg.device);
  if (ms_by_kind != nullptr && launches_by_kind != nullptr) {
    for (int k = 0; k < 8; ++k) { ms_by_kind[k] = 0.0; launches_by_kind[k] = 0; }
    if (h->ev_used > 0) CU_TRY(cudaEventSynchronize(h->ev_pool[h->ev_used - 1]));
    for (size_t i = 0; i + 1 < h->ev_used; ++i) {
      const int kind = h->ev_kind[i];
      if (kind == K_END) continue;
      float ms = 0.f;
      CU_TRY(cudaEventElapsedTime(&ms, h->ev_pool[i], h->ev_pool[i + 1]));
      ms_by_kind[kind] += ms;
      launches_by_kind[kind] += 1;
    }
  }
  h->ev_used = 0;
  h->profile = enable != 0;
  return XMC_OK;
}

int xmc_forward_logits(xmc_handle* h, const void* x, int32_t x_dtype, int32_t batch, void* out_bf16,
                       int64_t ld_out, int64_t n_out, void* stream) {
  if (h == nullptr || x == nullptr || out_bf16 == nullptr) return fail(XMC_ERR_INVALID, "null argument");
  if (h->w_ptrs.empty()) return fail(XMC_ERR_STATE, "xmc_bind_weights has not been called");
  if (x_dtype != XMC_DT_BF16 && x_dtype != XMC_DT_E4M3) return fail(XMC_ERR_INVALID, "embeddings must be bf16 or e4m3");
  if (batch <= 0 || batch > h->cfg.max_batch) return fail(XMC_ERR_INVALID, "batch %d outside [1, %d]", batch, h->cfg.max_batch);
  if (n_out <= 0 || n_out > h->total_rows || ld_out < n_out || (ld_out & 7) || ((uintptr_t)out_bf16 & 15u))
    return fail(XMC_ERR_INVALID, "bad output geometry (n_out %lld, ld_out %lld, rows %lld)", (long long)n_out, (long long)ld_out, (long long)h->total_rows);
  DeviceGuard guard(h->cfg.device);
  cudaStream_t st = (cudaStream_t)stream;
  const int d = h->cfg.dim, mode = h->cfg.mode;
  const bool fwd_fp8 = mode == XMC_MODE_FP8;
  // on CTA pairs (256 batch rows x 256 labels per pair, each CTA staging half of the tile's weight rows)
  // where both CTAs have batch rows to work on
  int max_pairs = 0;
  if (int rc = gradx_configure(h->sm_count, &max_pairs)) return rc;
  const bool pair = use_pairs(max_pairs) && batch > 128, sim = mode == XMC_MODE_SIMFP8;
  xmc::LogitsParams lp;
  lp.m_rows = pair ? 256 : 128;
  lp.x_rows = inference_rows(batch);
  lp.batch = batch;
  lp.n_mtiles = cdiv(batch, lp.m_rows);
  lp.lt = label_tiles(h, 256, 0, tiles_up_to(h, n_out));
  const int tiles = lp.n_mtiles * lp.lt.count;
  lp.div_mtiles = xmc::make_fastdiv(lp.n_mtiles, tiles);
  const bool split = sim && split_pays(h, tiles, max_pairs, pair), convert = sim && !split;
  CUtensorMap map_x;
  if (int rc = inference_operand(h, x, x_dtype, batch, split, lp.x_rows, &map_x, &lp.own_prep, st)) return rc;
  lp.w_maps = chunk_maps(h, convert ? (pair ? W_RAW128 : W_RAW256) : (pair ? W_ROWS128 : W_ROWS256));
  lp.k_steps = cdiv((long long)d * (fwd_fp8 || split ? 1 : 2), 128);
  lp.w_scale = h->cfg.w_scale;
  lp.x_scale = h->x_scale;
  lp.part_rows = x_rows_of(h);
  lp.x_wide = x_dtype == XMC_DT_E4M3 ? nullptr : h->x_wide;
  lp.out = reinterpret_cast<__nv_bfloat16*>(out_bf16);
  lp.ld_out = ld_out;
  lp.n_out = n_out;
  lp.status = h->status;
  // the output in boxes of 32 rows x 64 columns
  CUtensorMap map_out;
  if (int rc = make_map(&map_out, false, out_bf16, (uint64_t)n_out, (uint64_t)batch, (uint64_t)ld_out * 2, 64, 32)) return rc;
  mark(h, K_LOGITS, st);
  int rc;
#define XMC_LOGITS(PAIR_, FP8_, SIM_) launch_gemm<xmc::LogitsPolicy<FP8_, SIM_>, PAIR_>(map_x, map_x, lp, tiles, h->sm_count, st, 0, &map_out)
  if (split) rc = pair ? XMC_LOGITS(true, true, xmc::kSimSplit) : XMC_LOGITS(false, true, xmc::kSimSplit);
  else if (convert) rc = pair ? XMC_LOGITS(true, false, xmc::kSimConvert) : XMC_LOGITS(false, false, xmc::kSimConvert);
  else if (fwd_fp8) rc = pair ? XMC_LOGITS(true, true, xmc::kSimNone) : XMC_LOGITS(false, true, xmc::kSimNone);
  else rc = pair ? XMC_LOGITS(true, false, xmc::kSimNone) : XMC_LOGITS(false, false, xmc::kSimNone);
#undef XMC_LOGITS
  if (rc) return rc;
  mark(h, K_END, st);
  return XMC_OK;
}
int xmc_forward_topk(xmc_handle* h, const void* x, int32_t x_dtype, int32_t batch, int32_t k, int64_t n_out,
                     float* vals, int32_t* idx, void* stream) {
  if (h == nullptr || x == nullptr || vals == nullptr || idx == nullptr) return fail(XMC_ERR_INVALID, "null argument");
  if (h->w_ptrs.empty()) return fail(XMC_ERR_STATE, "xmc_bind_weights has not been called");
  if (x_dtype != XMC_DT_BF16 && x_dtype != XMC_DT_E4M3) return fail(XMC_ERR_INVALID, "embeddings must be bf16 or e4m3");
  if (batch <= 0 || batch > h->cfg.max_batch) return fail(XMC_ERR_INVALID, "batch %d outside [1, %d]", batch, h->cfg.max_batch);
  if (k <= 0 || k > 128) return fail(XMC_ERR_INVALID, "k must be in [1, 128], got %d", k);
  if (n_out <= 0 || n_out > h->total_rows) return fail(XMC_ERR_INVALID, "n_out %lld outside [1, %lld]", (long long)n_out, (long long)h->total_rows);
  DeviceGuard guard(h->cfg.device);
  cudaStream_t st = (cudaStream_t)stream;
  const int d = h->cfg.dim, mode = h->cfg.mode;
  const bool fwd_fp8 = mode == XMC_MODE_FP8;
  // CTA pairs where both CTAs have batch rows to work on
  int max_pairs = 0;
  if (int rc = gradx_configure(h->sm_count, &max_pairs)) return rc;
  const bool sim = mode == XMC_MODE_SIMFP8;
  const bool pair = use_pairs(max_pairs) && batch > 128;

  // Windows of label tiles: their logits live in G, whose size therefore bounds batch x window, and a merge follows
  // each.  Equal windows rather than full ones and a remainder.
  const int n_lt = tiles_up_to(h, n_out);
  const int64_t most = std::min<int64_t>((round_up(h->g_rows, 256) * h->bpad_max) / batch / 256, xmc::kTopkMaxGroups / 8);
  const int window = cdiv(n_lt, cdiv(n_lt, most));
  const int64_t ld_gmax = (int64_t)window * 8;

  if ((int64_t)batch * ld_gmax > h->topk_gmax_cap) {
    CU_TRY(cudaStreamSynchronize(st));
    if (h->topk_gmax) { cudaFree(h->topk_gmax); h->ws_bytes -= h->topk_gmax_cap * 2; h->topk_gmax = nullptr; h->topk_gmax_cap = 0; }
    // capacity x batch is about the size of G whatever the batch: one allocation serves every later call
    const int64_t want = std::max<int64_t>((int64_t)batch * ld_gmax, round_up(h->g_rows, 256) * h->bpad_max / 32);
    if (int rc = dev_alloc(h, (void**)&h->topk_gmax, (size_t)want * 2, false)) return rc;
    h->topk_gmax_cap = want;
  }
  if (h->topk_run == nullptr) {            // one allocation: all three are there or none
    if (int rc = dev_alloc(h, (void**)&h->topk_run, (size_t)h->bpad_max * (xmc::kTopkMaxK * 8 + 8), false)) return rc;
    h->topk_cnt = reinterpret_cast<int*>(h->topk_run + (size_t)h->bpad_max * xmc::kTopkMaxK);
    h->topk_thr = reinterpret_cast<float*>(h->topk_cnt + h->bpad_max);
  }
  {
    static std::atomic<uint64_t> configured{0};
    if (!((configured.load(std::memory_order_relaxed) >> (h->cfg.device & 63)) & 1ull)) {
      CU_TRY(cudaFuncSetAttribute(xmc::topk_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::topk_smem_bytes(xmc::kTopkMaxGroups)));
      configured.fetch_or(1ull << (h->cfg.device & 63));
    }
  }
  CUtensorMap map_x;
  int own_prep = 0;
  const bool split = sim && split_pays(h, cdiv(batch, pair ? 256 : 128) * n_lt, max_pairs, pair), convert = sim && !split;
  if (int rc = inference_operand(h, x, x_dtype, batch, split, inference_rows(batch), &map_x, &own_prep, st)) return rc;

  xmc::TopkMerge mp;
  mp.gmax = h->topk_gmax;
  mp.ld_gmax = ld_gmax;
  mp.z = h->G;
  mp.ld_z = (int64_t)window * 256;
  mp.chunk_groups = cdiv(h->rows_per_chunk, 256) * 8;
  mp.chunk_rows = (int)h->rows_per_chunk;
  mp.label0 = h->cfg.label_offset;
  mp.k = k;
  mp.run = h->topk_run;
  mp.run_cnt = h->topk_cnt;
  mp.thr = h->topk_thr;
  mp.out_val = vals;
  mp.out_idx = idx;
  xmc::TopkParams tp;
  tp.m_rows = pair ? 256 : 128;
  tp.x_rows = inference_rows(batch);
  tp.batch = batch;
  tp.n_mtiles = cdiv(batch, tp.m_rows);
  tp.div_mtiles = xmc::make_fastdiv(tp.n_mtiles, (long long)tp.n_mtiles * window);
  tp.w_maps = chunk_maps(h, convert ? (pair ? W_RAW128 : W_RAW256) : (pair ? W_ROWS128 : W_ROWS256));
  tp.n_out = n_out;
  tp.k_steps = cdiv((long long)d * (fwd_fp8 || split ? 1 : 2), 128);
  tp.w_scale = h->cfg.w_scale;
  tp.x_scale = h->x_scale;
  tp.part_rows = x_rows_of(h);
  tp.x_wide = x_dtype == XMC_DT_E4M3 ? nullptr : h->x_wide;
  tp.out = h->G;
  tp.ld_out = (int64_t)window * 256;
  tp.gmax = h->topk_gmax;
  tp.ld_gmax = ld_gmax;
  tp.status = h->status;
  // Where the first window's logits leave by boxes.  By threads / by boxes, us: simulated FP8 with converted weights, 1 171 872 x 128 at batch 48 94.7
  // and 95.6, 64 96.6 and 95.6, 100 107.4 and 102.0, 200 000 x 768 at 64 70.1 and 69.1, 160 95.9 and 82.1; FP8 1 171 872 x 128 at 64
  // 87.4 and 90.2, 100 97.1 and 96.2, 160 154 and 148, 200 000 x 768 at 100 47.2 and 47.7, 160 58.0 and 56.4; bf16 weights
  // 300 000 x 256 at 160 64.7 and 61.2, 100 000 x 768 at 300 71.6 and 77.6.  Simulated FP8 with
  // split embeddings 585 936 x 256 at 64 59.9 and 62.3, 100 67.1 and 67.1, 160 102.8 and 97.2, 320 003 x 384 at 49 43.9 and 44.2, 128 58.0 and 55.6.
  const bool boxes = sim ? batch > (split ? 64 : 48) : batch > 64 && (tp.k_steps <= 4 || (fwd_fp8 && batch > 128));
  CUtensorMap map_out;                                     // boxes of 32 rows x 32 columns
  if (boxes)
    if (int rc = make_map(&map_out, false, h->G, (uint64_t)tp.ld_out, (uint64_t)batch, (uint64_t)tp.ld_out * 2, 32, 32, SWIZZLE_64)) return rc;
  for (int t0 = 0; t0 < n_lt; t0 += window) {
    tp.after_prep = t0 == 0 ? 1 : 0;
    tp.own_prep = t0 == 0 ? own_prep : 0;
    tp.lt = label_tiles(h, 256, t0, std::min(window, n_lt - t0));
    tp.thr = t0 == 0 ? nullptr : h->topk_thr;
    const int tiles = tp.n_mtiles * tp.lt.count;
    mark(h, K_LOGITS, st);
    const bool box = t0 == 0 && boxes;
    const std::true_type yes;
    const std::false_type no;
    auto launch = [&](auto fp8_, auto sim_, auto pair_, auto box_) {
      using Policy = xmc::TopkPolicy<decltype(fp8_)::value, decltype(sim_)::value, decltype(box_)::value>;
      return launch_gemm<Policy, decltype(pair_)::value>(map_x, map_x, tp, tiles, h->sm_count, st, 0, boxes ? &map_out : nullptr);
    };
    auto by_pair = [&](auto fp8_, auto sim_) {
      if (pair) return box ? launch(fp8_, sim_, yes, yes) : launch(fp8_, sim_, yes, no);
      return box ? launch(fp8_, sim_, no, yes) : launch(fp8_, sim_, no, no);
    };
    const std::integral_constant<xmc::Simulated, xmc::kSimNone> none;
    const std::integral_constant<xmc::Simulated, xmc::kSimConvert> conv;
    const std::integral_constant<xmc::Simulated, xmc::kSimSplit> parts;
    const int rc = split ? by_pair(yes, parts) : convert ? by_pair(no, conv) : fwd_fp8 ? by_pair(yes, none) : by_pair(no, none);
    if (rc) return rc;
    mp.n_groups = tp.lt.count * 8;
    mp.first_group = t0 * 8;
    mp.first = t0 == 0 ? 1 : 0;
    mp.last = t0 + tp.lt.count == n_lt ? 1 : 0;
    mark(h, K_LOGITS, st);
    CU_TRY(launch_pdl(xmc::topk_merge_kernel, batch, xmc::kTopkThreads, xmc::topk_smem_bytes(mp.n_groups), st, mp));
  }
  mark(h, K_END, st);
  return XMC_OK;
}

// ---------------------------------------------------------------------------------------------
// Allocation-free contraction  C[m x n] = A^T B  (A given as [k x m] bf16, B as [k x n] bf16 or e4m3):
// the grad_X kernel with its split-K partial sums kept in a fixed device array owned by the library.
// ---------------------------------------------------------------------------------------------
namespace {
constexpr size_t kNoAllocFloats = 2u << 20;              // 8 MiB of partial sums
constexpr int kNoAllocMaxDevices = 64;
// [0, kNoAllocFloats): partial sums; then 4 ints of kernel status.  Every GPU that loads the library
// carries one copy until the process exits.
static __device__ __align__(256) float g_noalloc_scratch[kNoAllocFloats + 64];
// Device addresses of the array, one per device, filled on the first call for that device.  In host
// code the symbol itself is only a stand-in; the address a kernel can use comes from
// cudaGetSymbolAddress with the device current.
static std::atomic<float*> g_noalloc_ptr[kNoAllocMaxDevices];
}  // namespace

int xmc_large_k_matmul_noalloc(int32_t device, const void* a_bf16, const void* b, int32_t b_dtype,
                               int32_t k, int32_t m, int32_t n, float* c_f32, void* stream) {
  if (a_bf16 == nullptr || b == nullptr || c_f32 == nullptr) return fail(XMC_ERR_INVALID, "null argument");
  if (b_dtype != XMC_DT_BF16 && b_dtype != XMC_DT_E4M3) return fail(XMC_ERR_INVALID, "b must be bf16 or e4m3");
  if (k <= 0 || m <= 0 || n <= 0 || (m % 64) != 0 || (n % 64) != 0)
    return fail(XMC_ERR_INVALID, "need k > 0 and m, n positive multiples of 64 (got k %d, m %d, n %d)", k, m, n);
  if ((size_t)m * (size_t)n > kNoAllocFloats)
    return fail(XMC_ERR_INVALID, "m*n = %lld exceeds the built-in scratch of %lld floats (8 MiB): use the handle-based API",
                (long long)m * n, (long long)kNoAllocFloats);
  if (((uintptr_t)c_f32 & 15u) != 0 || ((uintptr_t)a_bf16 & 15u) != 0 || ((uintptr_t)b & 15u) != 0)
    return fail(XMC_ERR_INVALID, "a, b and c must be 16-byte aligned");
  if (device < 0 || device >= kNoAllocMaxDevices) return fail(XMC_ERR_INVALID, "device %d out of range", device);
  DeviceGuard guard(device);
  if (g_noalloc_ptr[device].load(std::memory_order_acquire) == nullptr) {
    // set-up, once per device, with that device current (the guard above)
    int cc_major = 0;
    CU_TRY(cudaDeviceGetAttribute(&cc_major, cudaDevAttrComputeCapabilityMajor, device));
    if (cc_major != 10) return fail(XMC_ERR_CUDA, "device %d is not sm_100", device);
    float* ptr = nullptr;
    CU_TRY(cudaGetSymbolAddress((void**)&ptr, g_noalloc_scratch));
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<true, false, 2>));
    CU_TRY(cudaFuncSetAttribute(xmc::gradx_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, xmc::kGxSmemBytes<false, false, 2>));
    // two threads racing through the set-up compute the same address; the publication itself is atomic
    g_noalloc_ptr[device].store(ptr, std::memory_order_release);
  }
  float* scratch = g_noalloc_ptr[device].load(std::memory_order_acquire);
  int* status = reinterpret_cast<int*>(scratch + kNoAllocFloats);
  int sm_count = 0;
  CU_TRY(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
  cudaStream_t st = (cudaStream_t)stream;
  const bool f8 = b_dtype == XMC_DT_E4M3;
  CUtensorMap map_a, map_b;
  if (int rc = make_map_blocked(&map_a, false, a_bf16, m, k, m, xmc::kGxRows, true)) return rc;
  if (int rc = make_map_blocked(&map_b, f8, b, n, k, n, xmc::kGxRows, !f8)) return rc;
  xmc::GxParams gp;
  gp.bpad = m;
  gp.d = n;
  gp.n_btiles = cdiv(m, 256);
  gp.n_dtiles = cdiv(n, 256);
  const int tiles = gp.n_btiles * gp.n_dtiles;
  int n_splits = std::max(1, sm_count / tiles);
  n_splits = (int)std::min<size_t>((size_t)n_splits, kNoAllocFloats / ((size_t)m * n));
  gp.total_ksteps = cdiv(k, xmc::kGxRows);
  n_splits = std::max(1, std::min(n_splits, gp.total_ksteps));
  gp.n_splits = n_splits;
  gp.w_maps = nullptr;
  gp.first_kstep = 0;
  gp.ksteps_per_chunk = gp.total_ksteps;
  gp.chain_ksteps = gp.total_ksteps;
  gp.accumulate = 0;            // every slot in use is fully overwritten: nothing has to start at zero
  gp.partial = scratch;
  gp.status = status;           // zero in the library image; set by a kernel that gave up a wait, read and
                                // cleared by xmc_noalloc_check
  if (f8) xmc::gradx_kernel<true><<<tiles * n_splits, xmc::kGxThreads, xmc::kGxSmemBytes<true, false, 2>, st>>>(map_a, map_b, gp);
  else xmc::gradx_kernel<false><<<tiles * n_splits, xmc::kGxThreads, xmc::kGxSmemBytes<false, false, 2>, st>>>(map_a, map_b, gp);
  CU_TRY(cudaGetLastError());
  const long long total = (long long)m * n;
  const int blocks = (int)std::min<long long>((total + 127) / 128, (long long)sm_count * 8);
  CU_TRY(launch_pdl(xmc::reduce_gradx_kernel, blocks, xmc::kReduceThreads, 0, st, (const float*)scratch, n_splits, m, m, n, 1.0f, c_f32,
                    (__nv_bfloat16*)nullptr, xmc::LossSum{nullptr, 0, nullptr}));
  return XMC_OK;
}

int xmc_noalloc_check(int32_t device, void* stream) {
  if (device < 0 || device >= kNoAllocMaxDevices) return fail(XMC_ERR_INVALID, "device %d out of range", device);
  float* scratch = g_noalloc_ptr[device].load(std::memory_order_acquire);
  if (scratch == nullptr) return XMC_OK;                 // no allocation-free call has run on this device yet
  DeviceGuard guard(device);
  cudaStream_t st = (cudaStream_t)stream;
  CU_TRY(cudaStreamSynchronize(st));
  int host[4] = {0, 0, 0, 0};                            // a stack array: this call allocates nothing either
  int* status = reinterpret_cast<int*>(scratch + kNoAllocFloats);
  CU_TRY(cudaMemcpy(host, status, sizeof(host), cudaMemcpyDeviceToHost));
  if (host[0] != xmc::DEV_OK) {
    CU_TRY(cudaMemset(status, 0, sizeof(host)));
    return fail(XMC_ERR_DEVICE_FLAG, "allocation-free contraction: device status %d (block %d, site %d)", host[0], host[1], host[2]);
  }
  return XMC_OK;
}

struct xmc_stager {
  int device = 0;
  cudaStream_t stream = nullptr;
  struct Slot {
    cudaEvent_t ready = nullptr, consumed = nullptr;
    bool filled = false, released = false;
  };
  std::vector<Slot> slots;
};

int xmc_stager_create(int32_t device, int32_t depth, xmc_stager** out) {
  if (out == nullptr || depth <= 0 || depth > 1024) return fail(XMC_ERR_INVALID, "bad argument");
  *out = nullptr;
  DeviceGuard guard(device);
  xmc_stager* s = new xmc_stager();
  s->device = device;
  s->slots.resize((size_t)depth);
  cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
  for (auto& slot : s->slots) {
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&slot.ready, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&slot.consumed, cudaEventDisableTiming);
  }
  if (e != cudaSuccess) {
    xmc_stager_destroy(s);
    return fail(XMC_ERR_CUDA, "stager: %s", cudaGetErrorString(e));
  }
  *out = s;
  return XMC_OK;
}

int xmc_stager_destroy(xmc_stager* s) {
  if (s == nullptr) return XMC_OK;
  DeviceGuard guard(s->device);
  if (s->stream) cudaStreamSynchronize(s->stream);
  for (auto& slot : s->slots) {
    if (slot.ready) cudaEventDestroy(slot.ready);
    if (slot.consumed) cudaEventDestroy(slot.consumed);
  }
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return XMC_OK;
}

int xmc_stager_put(xmc_stager* s, int32_t slot, const void* host_a, void* pinned_a, void* device_a, int64_t bytes_a,
                   const void* host_b, void* pinned_b, void* device_b, int64_t bytes_b) {
  if (s == nullptr || slot < 0 || (size_t)slot >= s->slots.size() || bytes_a < 0 || bytes_b < 0) return fail(XMC_ERR_INVALID, "bad argument");
  DeviceGuard guard(s->device);
  auto& sl = s->slots[(size_t)slot];
  if (sl.filled) CU_TRY(cudaEventSynchronize(sl.ready));
  sl.filled = true;
  if (bytes_a > 0) memcpy(pinned_a, host_a, (size_t)bytes_a);
  if (bytes_b > 0) memcpy(pinned_b, host_b, (size_t)bytes_b);
  if (sl.released) CU_TRY(cudaStreamWaitEvent(s->stream, sl.consumed, 0));
  if (bytes_a > 0) CU_TRY(cudaMemcpyAsync(device_a, pinned_a, (size_t)bytes_a, cudaMemcpyHostToDevice, s->stream));
  if (bytes_b > 0) CU_TRY(cudaMemcpyAsync(device_b, pinned_b, (size_t)bytes_b, cudaMemcpyHostToDevice, s->stream));
  CU_TRY(cudaEventRecord(sl.ready, s->stream));
  return XMC_OK;
}

int xmc_stager_get(xmc_stager* s, int32_t slot, void* stream) {
  if (s == nullptr || slot < 0 || (size_t)slot >= s->slots.size()) return fail(XMC_ERR_INVALID, "bad argument");
  DeviceGuard guard(s->device);
  CU_TRY(cudaStreamWaitEvent((cudaStream_t)stream, s->slots[(size_t)slot].ready, 0));
  return XMC_OK;
}

int xmc_stager_release(xmc_stager* s, int32_t slot, void* stream) {
  if (s == nullptr || slot < 0 || (size_t)slot >= s->slots.size()) return fail(XMC_ERR_INVALID, "bad argument");
  DeviceGuard guard(s->device);
  CU_TRY(cudaEventRecord(s->slots[(size_t)slot].consumed, (cudaStream_t)stream));
  s->slots[(size_t)slot].released = true;
  return XMC_OK;
}

int xmc_test_sigmoid(int32_t device, const void* in_bf16, void* out_bf16, int32_t n, void* stream) {
  if (in_bf16 == nullptr || out_bf16 == nullptr || n <= 0) return fail(XMC_ERR_INVALID, "bad argument");
  DeviceGuard guard(device);
  xmc::sigmoid_probe_kernel<<<cdiv(n, 256), 256, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const __nv_bfloat16*>(in_bf16), reinterpret_cast<__nv_bfloat16*>(out_bf16), n);
  CU_TRY(cudaGetLastError());
  return XMC_OK;
}

int xmc_test_gemm(int32_t device, int32_t layout, int32_t dtype, int32_t M, int32_t N, int32_t K,
                  const void* A, const void* B, float* D, void* stream) {
  if (A == nullptr || B == nullptr || D == nullptr || M <= 0 || N <= 0 || K <= 0) return fail(XMC_ERR_INVALID, "bad argument");
  const bool inject = (layout & 8) != 0;
  const bool pair = (layout & 4) != 0;
  layout &= ~12;
  if (layout < 0 || layout > 3) return fail(XMC_ERR_INVALID, "layout must be 0..3 (| 4 | 8)");
  if (pair && (layout & 1) != 0) return fail(XMC_ERR_INVALID, "CTA pairs take K-major operands");
  if (inject && ((layout & 1) != 0 || K < 2 * (dtype == XMC_DT_E4M3 ? 128 : 64)))
    return fail(XMC_ERR_INVALID, "the wait-limit test takes K-major operands with at least two k-steps");
  if ((layout & 1) == 1 && dtype != XMC_DT_BF16) return fail(XMC_ERR_INVALID, "MN-major test takes bf16");
  if (dtype != XMC_DT_BF16 && dtype != XMC_DT_E4M3) return fail(XMC_ERR_INVALID, "dtype");
  DeviceGuard guard(device);
  int cc_major = 0, sm_count = 0;
  CU_TRY(cudaDeviceGetAttribute(&cc_major, cudaDevAttrComputeCapabilityMajor, device));
  CU_TRY(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
  if (cc_major != 10) return fail(XMC_ERR_CUDA, "device is not sm_100");
  int* status = nullptr;
  CU_TRY(cudaMalloc((void**)&status, 16));
  CU_TRY(cudaMemset(status, 0, 16));
  cudaStream_t st = (cudaStream_t)stream;
  const bool f8 = dtype == XMC_DT_E4M3;
  CUtensorMap ma, mb;
  xmc::PlainParams p;
  p.M = M; p.N = N;
  p.n_ntiles = cdiv(N, 256);
  p.D = D;
  p.checksum_only = (layout & 2) ? 1 : 0;
  p.test_wait_limit = inject ? 2000000ll : 0;      // ~1 ms
  p.test_skip_tile = inject ? 0 : -1;
  layout &= 1;
  p.m_rows = pair ? 256 : 128;
  p.n_mtiles = cdiv(M, p.m_rows);
  p.status = status;
  int rc = XMC_OK;
  if (layout == 0) {
    if ((rc = make_map_kmajor(&ma, f8, A, K, M, K, 128))) { cudaFree(status); return rc; }
    // a CTA of a pair stages only its half of the B rows
    if ((rc = make_map_kmajor(&mb, f8, B, K, N, K, pair ? 128 : 256))) { cudaFree(status); return rc; }
    p.k_steps = cdiv((long long)K * (f8 ? 1 : 2), 128);
    const int tiles = p.n_mtiles * p.n_ntiles;
    if (pair) rc = f8 ? launch_gemm<xmc::PlainPolicy<true, false>, true>(ma, mb, p, tiles, sm_count, st)
                      : launch_gemm<xmc::PlainPolicy<false, false>, true>(ma, mb, p, tiles, sm_count, st);
    else rc = f8 ? launch_gemm<xmc::PlainPolicy<true, false>>(ma, mb, p, tiles, sm_count, st)
                 : launch_gemm<xmc::PlainPolicy<false, false>>(ma, mb, p, tiles, sm_count, st);
  } else {
    if ((rc = make_map_mnmajor(&ma, A, M, K, M))) { cudaFree(status); return rc; }
    if ((rc = make_map_mnmajor(&mb, B, N, K, N))) { cudaFree(status); return rc; }
    p.k_steps = cdiv(K, 64);
    rc = launch_gemm<xmc::PlainPolicy<false, true>>(ma, mb, p, p.n_mtiles * p.n_ntiles, sm_count, st);
  }
  if (rc == XMC_OK) {
    cudaError_t e = cudaStreamSynchronize(st);
    int host[4] = {0, 0, 0, 0};
    if (e == cudaSuccess) e = cudaMemcpy(host, status, 16, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) rc = fail(XMC_ERR_CUDA, "test gemm: %s", cudaGetErrorString(e));
    else if (host[0] != 0) rc = fail(XMC_ERR_DEVICE_FLAG, "test gemm: device status %d (block %d, site %d)", host[0], host[1], host[2]);
  }
  cudaFree(status);
  return rc;
}

}  // extern "C"


