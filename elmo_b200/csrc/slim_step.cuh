// The whole layer step for small batches (bf16 weights, e4m3 with real or simulated FP8 arithmetic) in ONE kernel: forward, loss
// gradient, grad_X and the fused weight update of a label tile while its weights are on the chip.
//
// With the three separate kernels (forward, grad_X, update) every weight is fetched three times by kernels that
// each ramp up and drain once per weight chunk; at batches up to 128 the contractions are so thin that this,
// not arithmetic, is what a step consists of.  Here a cluster of two CTAs takes tiles of 128 label rows and
// shares a tile twice over: by BATCH for the logits (each CTA multiplies the whole weight rows with its half of
// the batch and sends its half of G to the other through distributed shared memory), by FEATURES for the rest
// (each CTA updates, and accumulates grad_X for, its half of the 128-feature boxes).
//
// With stochastic rounding what bounds it is instruction issue: the arithmetic of the update (xmc_policies.cuh: 16 cycles per
// e4m3 weight and scheduler), beside which everything else is arranged to hide.  Rounded to nearest, and with bf16 weights,
// it is the chain of a tile, logits -> G -> the other CTA -> U -> update -> gx, of which as many links as fit are under way at a time.  The
// dispatch goes up to batch 128 because the grad_X accumulators of half the features, half a Z and the update's chunks
// then just fit into the 512 columns of TMEM.
//
// Every link of that chain has warps of its own.  (G made by the workers between two boxes, one warp for the MMAs of U and gx, one
// for Z's loads and MMAs cost a tile 5 to 30 %: sharing their schedulers with sixteen busy warps, such warps take ten cycles and
// more an instruction, and clock stamps showed the MMA warp of U and gx, 2 400 cycles a box, and the one of Z, 1 450, at the end
// of their tether, and 3 000 to 4 000 cycles of a worker's tile in G.)  Thirty-two warps leave 64 registers a thread, of
// which the others give the workers 16 each (setmaxnreg).  Before and now, us: e4m3 300 000 x 768 batch 8 214 and 200, 64 226 and
// 205, 128 303 and 282; 600 000 x 256 batch 8 182 and 166, 128 298 and 240; rounded to nearest 600 000 x 256 batch 16 155 and 116,
// 400 000 x 768 batch 64 211 and 182; a tenth of the rows compensated, 312 330 x 768 batch 128, in a loop at the power cap, 370 and 340; bf16 300 000 x
// 768 batch 128 403 and 380, 468 746 x 256 batch 128 263 and 195.  Where every cluster has a single tile it is launch and latency, and
// there the larger block costs narrow layers up to 0.6 us (6 000 x 64, batch 64 14.5 and 14.7, 9 000 x 256 16.9 and 17.4).
//
//   warp 0        Z[128 labels x nb/2] += W box . X box (K = 128 e4m3 or 64 bf16 features a box): tcgen05.mma
//   warp 1        U[128 labels x 2 uw]  = G . X^T chunk           (bf16, K = batch)
//   warp 2        loads of X^T chunks; once only where those of all the CTA's features fit
//   warp 3        stores updated boxes back
//   warps 4..11   Z -> sigmoid - y -> G (bf16, both CTAs' shared memory), as many tiles ahead as G has buffers; a row's batch columns
//                 in turns of sixteen
//   warps 12..27  update of the boxes in place, in two teams of eight warps that take one half of every box each; the old e4m3
//                 weights, in registers at that point, are written out as bf16 for gx on the way
//   warp 28       loads for Z (128 rows x 128 bytes of weights and X, a small ring); asks L2 for the weights of the tile after
//                 next
//   warp 29       gx[128 features x nb] += (old W box)^T . G      (bf16, K = 128 labels)
//                 gx of all the CTA's boxes stays in TMEM until the last tile; with bf16 weights, and where BOUND says so, the workers
//                 add it to the partial sums in memory every few tiles and it starts from zero (a long sum in the
//                 accumulator loses digits).  bf16 weights need no copy: gx is multiplied from the box itself, before the
//                 workers rewrite it in place
//   warp 30       loads of the boxes to be updated, once more (from L2)
//   warp 31       simulated FP8 with a wide row (PrepX): what warps 0 and 28 do otherwise
//
// No updated box can be stored before BOTH CTAs have multiplied the old weights into Z: U needs all of G.
//
// TMEM columns: boxes0 x nb for gx, z_bufs x nb / 2 for Z, u_bufs x 2 uw for U.
#pragma once
#include "gemm_engine.cuh"
#include "numerics.cuh"
#include "xmc_policies.cuh"

namespace xmc {

constexpr int kSlWorkers = 16, kSlGWarps = 8;
constexpr int kSlZLoader = 4 + kSlGWarps + kSlWorkers, kSlGxIssuer = kSlZLoader + 1, kSlWLoader = kSlZLoader + 2;     // (the last warp: see SPLIT)
constexpr int kSlThreads = 32 * (kSlZLoader + 4);
// Registers a thread: as launched, what the register file holds for so many threads, and as the warpgroups share them
// out.
constexpr int kSlLaunchRegs = 65536 / kSlThreads / 8 * 8;
constexpr int kSlRoleRegs = 40, kSlLoaderRegs = 40;
// Compensated rows take more of a worker than 80: 312 330 x 768 batch 128, in a loop at the power cap, 344 and 340 us; G's warps can do with 40
// unless there is the loss to sum up.
__host__ __device__ constexpr int slim_g_regs(bool kahan) { return kahan ? 40 : 56; }
__host__ __device__ constexpr int slim_worker_regs(bool kahan) { return kahan ? 88 : 80; }
constexpr int slim_regs(bool kahan) {
  return 128 * (kSlRoleRegs + kSlGWarps / 4 * slim_g_regs(kahan) + kSlWorkers / 4 * slim_worker_regs(kahan) + kSlLoaderRegs);
}
static_assert(slim_regs(false) <= kSlThreads * kSlLaunchRegs && slim_regs(true) <= kSlThreads * kSlLaunchRegs,
              "more registers than the block is launched with: the warps that ask for them would wait for good");
constexpr int kSlBox = 128 * 128;               // one weight box: 128 rows x 128 bytes (features)
constexpr int kSlStaging = 2;
constexpr int kSlMaxZ = 4, kSlMaxW = 3, kSlMaxXt = 2, kSlMaxG = 3;

struct SlimParams {
  const CUtensorMap* w_maps;       // one per weight chunk: boxes of 128 rows x 128 bytes, 128-byte swizzle (device memory)
  int n_tiles;
  FastDiv div_tpc;                 // label tiles per chunk
  int rows_full, rows_last;        // label rows of every chunk but the last, of the last
  int n_chunks;
  int bkt_per_chunk;               // buckets (128 labels) per chunk
  int batch, nb;                   // batch rows; padded to a multiple of 32 (<= 128)
  int n_boxes;                     // 128-feature boxes of a row; CTA 0 of a cluster owns the first (n_boxes + 1) / 2
  int uw;                          // features per team in an update chunk: 64, or 32 where TMEM is short
  int u_bufs;                      // update chunks in TMEM at a time
  int z_bufs;                      // accumulators for Z: 2 where TMEM has room
  int z_stages, w_slots, xt_stages;
  int g_bufs;                      // G of so many tiles in shared memory
  int s_bufs;                      // e4m3: copies of old weights
  int gx_mask;                     // bf16: tiles that a grad_X accumulator sums up before it is added to `partial`, a power of two, minus one
  float w_scale;
  const float* x_scale;            // split embeddings: see FwdParams
  int part_rows;
  const uint8_t* x_wide;
  const int* bucket_off;
  const uint32_t* bucket_ent;
  double* loss_partial;            // [gridDim.x * kSlGWarps] or nullptr
  float* partial;                  // [clusters][nb][d]
  UpdParams upd;                   // kahan rows, learning rate, random stream; elem0 = element index of row 0 of chunk 0
  int* status;
  int gx_tiles;                    // BOUND: tiles that a grad_X accumulator sums up at most
};

struct SlimShared {
  uint64_t zf[kSlMaxZ], ze[kSlMaxZ];      // Z ring
  uint64_t z_full[2], z_empty[2];
  uint64_t g_ready[kSlMaxG], g_empty[kSlMaxG];        // G: own warps and the peer's bytes / the MMAs of both CTAs have read it
  uint64_t xf[kSlMaxXt], xe[kSlMaxXt];          // X^T chunks
  uint64_t wf[kSlMaxW], wd[kSlMaxW], we[kSlMaxW];   // weight boxes: landed, rewritten (and copied), stored
  uint64_t uf[2], ue[2];                        // update chunks
  uint64_t se[kSlStaging];                      // e4m3: the copy of the old weights has been multiplied
  uint64_t gf[kSlMaxW];                         // bf16: the box itself has been
  uint64_t gx_full;
  uint32_t tmem_base;
  Ctl ctl;
  alignas(16) float x_scale[64];                // split embeddings: of this CTA's half of the batch
};

__host__ __device__ constexpr int slim_k_blocks(int nb) { return (nb + 63) / 64; }
__host__ __device__ constexpr int slim_smem_bytes(bool w8, bool split, int nb, int uw, int z_stages, int w_slots, int xt_stages, int g_bufs, int s_bufs) {
  return z_stages * (kSlBox + (split ? 2 : 1) * nb * 64) + w_slots * (w8 ? kSlBox : 2 * kSlBox) + (w8 ? s_bufs * 2 * kSlBox : 0) + g_bufs * slim_k_blocks(nb) * kSlBox +
         xt_stages * slim_k_blocks(nb) * uw * 256 + kSlGWarps * 256 + (int)sizeof(SlimShared);
}

// 4 x 4 words of four neighbouring lanes: word k of lane j becomes word j of lane k
__device__ __forceinline__ void transpose4(uint32_t* v, int lane) {
#pragma unroll
  for (int m = 1; m <= 2; m <<= 1) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k & m) continue;
      const uint32_t got = __shfl_xor_sync(0xffffffffu, lane & m ? v[k] : v[k | m], m);
      if (lane & m) v[k] = got;
      else v[k | m] = got;
    }
  }
}

// Positives of a bucket among the label rows 32 q + [0, 32) and the batch columns b0 + [0, nz), nz <= 64: lane i gets the columns of
// row 32 q + i, a bit each; mrow: the warp's 64 words of shared memory.  Four entries a lane are under way at a time, without a
// branch for each: with one entry a turn the popular labels of 6 000 x 768 at batch 128, 20 positives a row, were 31 -> 39 us.
__device__ __forceinline__ uint2 slim_positives(const uint32_t* __restrict__ ents, int beg, int end, int q, int b0, int nz, uint32_t mrow) {
  const int lane = threadIdx.x & 31;
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(mrow + 4u * (uint32_t)lane), "r"(0u) : "memory");
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(mrow + 128u + 4u * (uint32_t)lane), "r"(0u) : "memory");
  __syncwarp();
  for (int e0 = beg + lane; e0 < end; e0 += 128) {
    uint32_t ent[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) ent[u] = e0 + 32 * u < end ? ents[e0 + 32 * u] : 0xFFFFFFFFu;   // no row of any tile
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t lrow = ent[u] >> 16, c = (ent[u] & 0xFFFFu) - (uint32_t)b0;
      const uint32_t in = (uint32_t)((lrow >> 5) == (uint32_t)q) & (uint32_t)(c < (uint32_t)nz);
      asm volatile("{.reg .pred p; setp.ne.u32 p, %2, 0; @p red.shared.or.b32 [%0], %1;}" ::"r"(mrow + (c & 32u) * 4u + 4u * (lrow & 31u)),
                   "r"(1u << (c & 31u)), "r"(in) : "memory");
    }
  }
  __syncwarp();
  uint2 bits;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(bits.x) : "r"(mrow + 4u * (uint32_t)lane) : "memory");
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(bits.y) : "r"(mrow + 128u + 4u * (uint32_t)lane) : "memory");
  __syncwarp();
  return bits;
}

// What compensates the first rows of chunk 0.  A kernel for either type: with both in one, bf16 terms took 1 to 4 % longer.
enum KahanTerms { kKahanNone, kKahanBf16, kKahanE5m2 };

// U_WAITS: with a box's first chunk of U everything the workers need for it is there, so they wait for U alone; else each worker waits
// for the weights and, before it writes, for their copy's buffer, and U may run ahead of them.  The workers' waits cost 2 to 5 % (300 000 x
// 768, batch 8 212 -> 201 us without), but from batch 65 on, where rings are short and chunks half a box, U held up by
// the weights costs more (300 000 x 768, batch 128 299 -> 282; 200 000 x 384 148 -> 138).
// SPLIT: simulated FP8, embeddings in two parts, with a wide row in four (PrepX).  (Three kernels and this one, us: 131 072 x 768 batch 16 157 and 100 -- 145 with
// split embeddings there too --, 200 000 x 1 024 rounded to nearest batch 16 253 and 140, 4 001 x 64 batch 16 22.7 and 13.1.)
// BOUND: sums of grad_X over e4m3 weights that may end before the last tile (gx_tiles): in the kernels that took over from three with
// shorter ones, layers rounded to nearest and simulated FP8, the latter only where they would be longer.  The workers' loop is
// where there is the least room: the loop around it costs 5 to 9 % of simulated FP8 at batch 64, ended sums or not (600 000 x 256 194 -> 206
// us), up to 8 % of stochastic rounding, 1 % of rounding to nearest; with the end of a sum in the middle of the loop, or
// added by the warps of G, up to 10 % more.
template <bool W8, bool SR, bool LOSS, KahanTerms KAHAN, bool U_WAITS, bool SPLIT = false, bool BOUND = false>
__global__ void __launch_bounds__(kSlThreads, 1)
slim_step_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_xt,
                 const __grid_constant__ SlimParams p) {
  using Upd = UpdPolicy<W8, SR, !W8, false, KAHAN != kKahanNone>;
  constexpr int kWSlot = W8 ? kSlBox : 2 * kSlBox;               // 128 features of 128 rows
  constexpr bool kLateWait = KAHAN == kKahanNone;                // (compensated rows, 300 000 x 384 batch 96: at the start of a box 219 us, late 226)
  constexpr int kZFeatures = W8 ? 128 : 64;                      // features of a Z box: 128 bytes of a row
  static_assert(!BOUND || (W8 && KAHAN == kKahanNone), "bf16 weights end their sums box by box, compensated rows none");
  extern __shared__ __align__(1024) uint8_t smem[];
  const int nb = p.nb, nz = nb >> 1, nkb = slim_k_blocks(nb), d = p.upd.d;
  static_assert(W8 || !SPLIT, "the parts are FP8 operands");
  const int z_stage = kSlBox + (SPLIT ? 2 : 1) * nz * 128, xt_stage = nkb * p.uw * 256;
  uint8_t* smem_z = smem;                                        // [stage][W box | X box, of split embeddings two]
  uint8_t* smem_w = smem_z + p.z_stages * z_stage;               // [slot][128 rows][128 B], bf16: two blocks of 64 features
  uint8_t* smem_s = smem_w + p.w_slots * kWSlot;                 // e4m3: [buffer][2 blocks of 64 features][128 rows][128 B]
  uint8_t* smem_g = smem_s + (W8 ? p.s_bufs * 2 * kSlBox : 0);            // [buffer][blocks of 64 batch rows][128 labels][128 B]
  uint8_t* smem_xt = smem_g + p.g_bufs * nkb * kSlBox;               // [stage][blocks of 64 batch rows][2 uw features][128 B]
  uint32_t* smem_m = reinterpret_cast<uint32_t*>(smem_xt + p.xt_stages * xt_stage);    // [G warp][2 x 32 columns][32 rows]
  SlimShared& sh = *reinterpret_cast<SlimShared*>(smem_m + kSlGWarps * 64);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int worker = (int)(blockIdx.x >> 1), n_workers = (int)(gridDim.x >> 1);
  const int boxes0 = (p.n_boxes + 1) >> 1;
  const int my_boxes = rank == 0 ? boxes0 : p.n_boxes - boxes0, box0 = rank == 0 ? 0 : boxes0;
  const int subs = 64 / p.uw;                                    // chunks per box
  const int n_iter = (p.n_tiles - worker + n_workers - 1) / n_workers;
  const uint32_t z_col = (uint32_t)(boxes0 * nb), u_col = z_col + (uint32_t)(p.z_bufs * nz);

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSlMaxZ; ++i) { mbar_init(smem_u32(&sh.zf[i]), 1); mbar_init(smem_u32(&sh.ze[i]), 1); }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sh.z_full[i]), 1);
      mbar_init(smem_u32(&sh.z_empty[i]), kSlGWarps);
    }
    for (int i = 0; i < kSlMaxG; ++i) { mbar_init(smem_u32(&sh.g_ready[i]), kSlGWarps); mbar_init(smem_u32(&sh.g_empty[i]), 4); }
    for (int i = 0; i < kSlMaxXt; ++i) { mbar_init(smem_u32(&sh.xf[i]), 1); mbar_init(smem_u32(&sh.xe[i]), 1); }
    for (int i = 0; i < kSlMaxW; ++i) {
      mbar_init(smem_u32(&sh.wf[i]), 1);
      mbar_init(smem_u32(&sh.wd[i]), kSlWorkers);
      mbar_init(smem_u32(&sh.we[i]), 1);
      mbar_init(smem_u32(&sh.gf[i]), 1);
    }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&sh.uf[i]), 1); mbar_init(smem_u32(&sh.ue[i]), kSlWorkers); }
    for (int i = 0; i < kSlStaging; ++i) mbar_init(smem_u32(&sh.se[i]), 1);
    mbar_init(smem_u32(&sh.gx_full), 1);
    sh.ctl.abort = 0;
    sh.ctl.limit = kWaitLimitCycles;
    fence_barrier_init();
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&map_xt);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&sh.tmem_base), kTmemCols);
    tmem_relinquish();
  }
  // the warps that load or store weights
  if (warp == 3 || warp == kSlZLoader || warp == kSlWLoader || (SPLIT && warp == kSlWLoader + 1)) tensormap_acquire(p.w_maps, 0, p.n_chunks - 1);
  pdl_launch_dependents();
  tc_fence_before();
  cluster_sync_all();                     // both CTAs' barriers exist before anything remote happens
  pdl_wait();
  tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;

  // tile -> chunk and first row within it
  auto tile_at = [&](int i, int& ci, int& row0) {
    const int tile = worker + i * n_workers;
    ci = fast_div(tile, p.div_tpc);
    row0 = (tile - ci * p.div_tpc.d) * 128;
  };

  const bool xt_kept = my_boxes * subs <= p.xt_stages;           // X^T of all the CTA's features fits: fetched once
  const uint32_t xt_ring = (uint32_t)(xt_kept ? my_boxes * subs : p.xt_stages);
  auto g_there = [&](uint32_t gb, uint32_t gph) {
    if (!mbar_wait_warp(smem_u32(&sh.g_ready[gb]), gph, &sh.ctl, p.status, 813)) return false;
    mbar_acquire_cluster(smem_u32(&sh.g_ready[gb]), gph);
    fence_proxy_async();                            // the peer's half of G came by generic-proxy stores
    return true;
  };
  if (warp < 4) warp_regs<kSlLaunchRegs, kSlRoleRegs>();
  if (warp >= kSlZLoader) warp_regs<kSlLaunchRegs, kSlLoaderRegs>();
  if (warp >= kSlZLoader) {
    // ------------------------------ loads for Z ------------------------------
    if (warp == kSlZLoader) {
      const uint32_t z0 = smem_u32(smem_z), zf0 = smem_u32(&sh.zf[0]), ze0 = smem_u32(&sh.ze[0]);
      const int n_zboxes = (d + kZFeatures - 1) / kZFeatures;
      uint32_t s = 0, ph = 1u;
      bool ok = true;
      // whether a row is wide is looked at when the first tile's first parts are on their way
      [[maybe_unused]] const uint32_t wide = SPLIT ? wide_rows(p.x_wide, p.batch, 0) : 0u;
      for (int i = 0; ok && i < n_iter; ++i) {
        int ci, row0;
        tile_at(i, ci, row0);
        if (i + 2 < n_iter) {
          // the CTAs of a cluster fetch the same boxes: each asks L2 for every other one
          int cn, rn;
          tile_at(i + 2, cn, rn);
          if (elect_one())
            for (int k = (int)rank; k < n_zboxes; k += 2) tma_prefetch_2d(p.w_maps + cn, k * kZFeatures, rn);
          __syncwarp();
        }
        const CUtensorMap* wm = p.w_maps + ci;
        for (int k = 0; k < n_zboxes; ++k) {
          if (!mbar_wait_warp(ze0 + 8u * s, ph, &sh.ctl, p.status, 800)) { ok = false; break; }
          if (elect_one()) {
            const uint32_t bar = zf0 + 8u * s, dst = z0 + s * (uint32_t)z_stage;
            mbar_arrive_expect_tx(bar, (uint32_t)z_stage);
            tma_load_2d(dst, wm, bar, k * kZFeatures, row0);
            tma_load_2d(dst + kSlBox, &map_x, bar, k * kZFeatures, (int)rank * nz);
            if constexpr (SPLIT) tma_load_2d(dst + kSlBox + (uint32_t)nz * 128u, &map_x, bar, k * kZFeatures, (int)rank * nz + p.part_rows);
          }
          __syncwarp();
          if (++s == (uint32_t)p.z_stages) { s = 0; ph ^= 1u; }
        }
        if (SPLIT && i == 0 && __any_sync(0xffffffffu, wide != 0u)) break;       // the last warp goes on
      }
    } else if (warp == kSlGxIssuer) {
      // ------------------------------ MMA issuer for gx ------------------------------
      // From the old weights: the e4m3 boxes' copies, once the workers have made them, or the bf16 boxes themselves, before
      // the workers rewrite them.
      constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
      const uint32_t idesc_g = make_idesc(128, (uint32_t)nb, 1u, 1u, 1u, 1u);
      // both operands MN-major: blocks of 64 elements kSlBox apart, one MMA eats 16 label rows = 2048 B
      const uint32_t g_lo0 = smem_desc_lo(smem_u32(smem_g), kSlBox), w_lo0 = smem_desc_lo(smem_u32(W8 ? smem_s : smem_w), kSlBox);
      const uint32_t g_step = (uint32_t)(nkb * kSlBox) >> 4;
      uint32_t ws = 0, wph = 0, ss = 0, gb = 0, gph = 0;
      [[maybe_unused]] uint32_t ds = 0, dph = 0;                 // bf16: the slot that this box had a tile ago
      bool ok = true;
      auto tiles = [&](int first, int end) {
        for (int i = first; ok && i < end; ++i) {
          if (!g_there(gb, gph)) {
            if (BOUND) ok = false;
            break;
          }
          const bool fresh = W8 ? i == first : (i & p.gx_mask) == 0;       // a sum begins
          for (int bx = 0; bx < my_boxes; ++bx) {
            if (!mbar_wait_warp(smem_u32(W8 ? &sh.wd[ws] : &sh.wf[ws]), wph, &sh.ctl, p.status, 812)) { ok = false; break; }
            if constexpr (!W8) {
              // The sum before has to be out of TMEM: the workers have left the box of the tile before.  With as many
              // boxes a tile as slots, or more, this box's slot has shown it.
              if (i > 0 && my_boxes < p.w_slots) {
                if (fresh && !mbar_wait_warp(smem_u32(&sh.wd[ds]), dph, &sh.ctl, p.status, 818)) { ok = false; break; }
                if (++ds == (uint32_t)p.w_slots) { ds = 0; dph ^= 1u; }
              }
            }
            tc_fence_after();
            if (elect_one()) {
              const uint32_t a = w_lo0 + (W8 ? ss : ws) * (2u * kSlBox >> 4), b = g_lo0 + gb * g_step, dt = tmem_base + (uint32_t)(bx * nb);
              umma_f16_lohi(dt, a, b, desc_hi, idesc_g, fresh ? 0u : 1u);
#pragma unroll
              for (uint32_t u = 1; u < 8; ++u) umma_f16_lohi(dt, a + 128u * u, b + 128u * u, desc_hi, idesc_g, 1u);
              umma_commit(smem_u32(W8 ? &sh.se[ss] : &sh.gf[ws]));
            }
            __syncwarp();
            if (++ss == (uint32_t)p.s_bufs) ss = 0;
            if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
          }
          if (ok && i + p.g_bufs < n_iter && elect_one()) umma_commit_both(smem_u32(&sh.g_empty[gb]));
          __syncwarp();
          if (++gb == (uint32_t)p.g_bufs) { gb = 0; gph ^= 1u; }
        }
        if (ok && elect_one()) umma_commit(smem_u32(&sh.gx_full));
        __syncwarp();
      };
      if constexpr (BOUND) {
        for (int i = 0; ok && i < n_iter; i += p.gx_tiles) tiles(i, min(n_iter, i + p.gx_tiles));
      } else {
        tiles(0, n_iter);
      }
    } else if (warp == kSlWLoader) {
      // ------------------------------ loads of the boxes to be updated ------------------------------
      uint32_t ws = 0, wph = 1u;
      bool ok = true;
      for (int i = 0; ok && i < n_iter; ++i) {
        int ci, row0;
        tile_at(i, ci, row0);
        const CUtensorMap* wm = p.w_maps + ci;
        for (int bx = 0; bx < my_boxes; ++bx) {
          if (!mbar_wait_warp(smem_u32(&sh.we[ws]), wph, &sh.ctl, p.status, 820)) { ok = false; break; }
          if (elect_one()) {
            const uint32_t bar = smem_u32(&sh.wf[ws]);
            mbar_arrive_expect_tx(bar, kWSlot);
            tma_load_2d(smem_u32(smem_w + ws * kWSlot), wm, bar, (box0 + bx) * 128, row0);
            if constexpr (!W8) tma_load_2d(smem_u32(smem_w + ws * kWSlot + kSlBox), wm, bar, (box0 + bx) * 128 + 64, row0);
          }
          __syncwarp();
          if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
        }
      }
    } else if constexpr (SPLIT) {
      // ------------------------------ Z of wide rows ------------------------------
      // Loads, but for the first tile's first parts, and MMAs, over the features twice.  (By the two warps that do it for narrow
      // rows, in one loop or in loops of their own, those paid for it: 150 000 x 128 rounded to nearest, batch 33 45.5 and 47.4 us.)
      if (__any_sync(0xffffffffu, wide_rows(p.x_wide, p.batch, 0) != 0u)) {
        constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
        const uint32_t idesc = make_idesc(128, (uint32_t)nz, 0u, 0u, 0u, 0u), idesc_2 = make_idesc(128, (uint32_t)nz, 0u, 1u, 0u, 0u);
        const int n_zboxes = (d + kZFeatures - 1) / kZFeatures;
        const uint32_t z0 = smem_u32(smem_z), zf0 = smem_u32(&sh.zf[0]), ze0 = smem_u32(&sh.ze[0]), z_lo0 = smem_desc_lo(z0, 16);
        uint32_t ls = 0, lph = 1u, s = 0, ph = 0, zb = 0, zph = 1u;
        int li = 0, lk = 0, i = 0, k = 0;                        // tile and box of the next load, of the next MMA
        bool ok = true;
        while (ok && i < n_iter) {
          // as many loads ahead as there are stages
          for (int ahead = (li - i) * 2 * n_zboxes + lk - k; ok && li < n_iter && ahead < p.z_stages; ++ahead) {
            if (li > 0 || lk >= n_zboxes) {
              int ci, row0;
              tile_at(li, ci, row0);
              if (!mbar_wait_warp(ze0 + 8u * ls, lph, &sh.ctl, p.status, 800)) { ok = false; break; }
              if (elect_one()) {
                const uint32_t bar = zf0 + 8u * ls, dst = z0 + ls * (uint32_t)z_stage;
                mbar_arrive_expect_tx(bar, (uint32_t)z_stage);
                const int f = (lk < n_zboxes ? lk : lk - n_zboxes) * kZFeatures, x_row = (int)rank * nz + (lk < n_zboxes ? 0 : 2 * p.part_rows);
                tma_load_2d(dst, p.w_maps + ci, bar, f, row0);
                tma_load_2d(dst + kSlBox, &map_x, bar, f, x_row);
                tma_load_2d(dst + kSlBox + (uint32_t)nz * 128u, &map_x, bar, f, x_row + p.part_rows);
              }
              __syncwarp();
            }
            if (++ls == (uint32_t)p.z_stages) { ls = 0; lph ^= 1u; }
            if (++lk == 2 * n_zboxes) { lk = 0; ++li; }
          }
          if (!ok || (k == 0 && !mbar_wait_warp(smem_u32(&sh.z_empty[zb]), zph, &sh.ctl, p.status, 801)) ||
              !mbar_wait_warp(zf0 + 8u * s, ph, &sh.ctl, p.status, 802)) break;
          tc_fence_after();
          if (elect_one()) {
            const uint32_t a = z_lo0 + s * ((uint32_t)z_stage >> 4), b = a + (kSlBox >> 4), b2 = b + (uint32_t)nz * 8u;
            const uint32_t d_tmem = tmem_base + z_col + zb * (uint32_t)nz;
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) umma_f8_lohi(d_tmem, a + 2u * u, b2 + 2u * u, desc_hi, idesc_2, (k | (int)u) ? 1u : 0u);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) umma_f8_lohi(d_tmem, a + 2u * u, b + 2u * u, desc_hi, idesc, 1u);
            umma_commit(ze0 + 8u * s);
            if (k + 1 == 2 * n_zboxes) umma_commit(smem_u32(&sh.z_full[zb]));
          }
          __syncwarp();
          if (++s == (uint32_t)p.z_stages) { s = 0; ph ^= 1u; }
          if (++k == 2 * n_zboxes) {
            k = 0;
            ++i;
            if (++zb == (uint32_t)p.z_bufs) { zb = 0; zph ^= 1u; }
          }
        }
      }
    }
  } else if (warp == 0) {
    // ------------------------------ MMA issuer for Z ------------------------------
    constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
    constexpr uint32_t kFmt = W8 ? 0u : 1u;                      // e4m3, bf16
    const uint32_t idesc = make_idesc(128, (uint32_t)nz, kFmt, kFmt, 0u, 0u);
    const uint32_t zf0 = smem_u32(&sh.zf[0]), ze0 = smem_u32(&sh.ze[0]), z_lo0 = smem_desc_lo(smem_u32(smem_z), 16);
    const int n_zboxes = (d + kZFeatures - 1) / kZFeatures;
    uint32_t s = 0, ph = 0, zb = 0, zph = 1u;
    bool ok = true;
    if constexpr (SPLIT) ok = !__any_sync(0xffffffffu, wide_rows(p.x_wide, p.batch, 0) != 0u);       // else the last warp does it
    for (int i = 0; ok && i < n_iter; ++i) {
      if (!mbar_wait_warp(smem_u32(&sh.z_empty[zb]), zph, &sh.ctl, p.status, 801)) break;
      const uint32_t d_tmem = tmem_base + z_col + zb * (uint32_t)nz;
      for (int k = 0; k < n_zboxes; ++k) {
        if (!mbar_wait_warp(zf0 + 8u * s, ph, &sh.ctl, p.status, 802)) { ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a = z_lo0 + s * ((uint32_t)z_stage >> 4), b = a + (kSlBox >> 4);
          if constexpr (SPLIT) {
            const uint32_t b2 = b + (uint32_t)nz * 8u, idesc_2 = make_idesc(128, (uint32_t)nz, 0u, 1u, 0u, 0u);     // e4m3 by e5m2
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) umma_f8_lohi(d_tmem, a + 2u * u, b2 + 2u * u, desc_hi, idesc_2, (k | (int)u) ? 1u : 0u);
          }
#pragma unroll
          for (uint32_t u = 0; u < 4; ++u) {
            if constexpr (W8) umma_f8_lohi(d_tmem, a + 2u * u, b + 2u * u, desc_hi, idesc, SPLIT || (k | (int)u) ? 1u : 0u);
            else umma_f16_lohi(d_tmem, a + 2u * u, b + 2u * u, desc_hi, idesc, (k | (int)u) ? 1u : 0u);
          }
          umma_commit(ze0 + 8u * s);
          if (k + 1 == n_zboxes) umma_commit(smem_u32(&sh.z_full[zb]));
        }
        __syncwarp();
        if (++s == (uint32_t)p.z_stages) { s = 0; ph ^= 1u; }
      }
      if (++zb == (uint32_t)p.z_bufs) { zb = 0; zph ^= 1u; }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer for U ------------------------------
    constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
    const uint32_t idesc_u = make_idesc(128, 2u * (uint32_t)p.uw, 1u, 1u, 0u, 0u);
    const uint32_t g_lo0 = smem_desc_lo(smem_u32(smem_g), 16), xt_lo0 = smem_desc_lo(smem_u32(smem_xt), 16);
    const uint32_t g_step = (uint32_t)(nkb * kSlBox) >> 4, xt_blk = (uint32_t)p.uw * 16u;
    uint32_t xs = 0, xph = 0, ub = 0, uph = 1u, gb = 0, gph = 0, ws = 0, wph = 0, ss = 0, sph = 1u;
    bool ok = true;
    for (int i = 0; ok && i < n_iter; ++i) {
      if (!g_there(gb, gph)) break;
      for (int c = 0; c < my_boxes * subs; ++c) {
        if (!mbar_wait_warp(smem_u32(&sh.xf[xs]), xph, &sh.ctl, p.status, 814) ||
            !mbar_wait_warp(smem_u32(&sh.ue[ub]), uph, &sh.ctl, p.status, 815)) { ok = false; break; }
        if (U_WAITS && (subs == 1 || (c & 1) == 0)) {
          // the weights have landed, and the buffer of their copy is free; bf16: the old weights have been multiplied
          if constexpr (W8) {
            if (!mbar_wait_warp(smem_u32(&sh.wf[ws]), wph, &sh.ctl, p.status, 816) ||
                !mbar_wait_warp(smem_u32(&sh.se[ss]), sph, &sh.ctl, p.status, 817)) { ok = false; break; }
            if (++ss == (uint32_t)p.s_bufs) { ss = 0; sph ^= 1u; }
          } else {
            if (!mbar_wait_warp(smem_u32(&sh.gf[ws]), wph, &sh.ctl, p.status, 816)) { ok = false; break; }
          }
          if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
        }
        tc_fence_after();
        if (elect_one()) {
          uint32_t a = g_lo0 + gb * g_step, b = xt_lo0 + xs * ((uint32_t)xt_stage >> 4);
          const uint32_t dt = tmem_base + u_col + ub * 2u * (uint32_t)p.uw;
          for (int kb = 0; kb < nb; kb += 64, a += kSlBox >> 4, b += xt_blk) {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
              if (u < 2 || kb + 32 < nb) umma_f16_lohi(dt, a + 2u * u, b + 2u * u, desc_hi, idesc_u, (kb | (int)u) ? 1u : 0u);
            }
          }
          umma_commit(smem_u32(&sh.uf[ub]));
          if (!xt_kept) umma_commit(smem_u32(&sh.xe[xs]));
        }
        __syncwarp();
        if (++xs == xt_ring) {
          xs = 0;
          if (!xt_kept) xph ^= 1u;
        }
        if (++ub == (uint32_t)p.u_bufs) { ub = 0; uph ^= 1u; }
      }
      // (not for the last tiles: nobody waits for those buffers again, and a late arrival at the peer could meet
      // the shared memory of the next kernel there)
      if (ok && i + p.g_bufs < n_iter && elect_one()) umma_commit_both(smem_u32(&sh.g_empty[gb]));
      __syncwarp();
      if (++gb == (uint32_t)p.g_bufs) { gb = 0; gph ^= 1u; }
    }
  } else if (warp == 2) {
    // ------------------------------ loads of X^T ------------------------------
    uint32_t xs = 0, xph = 1u;
    bool ok = true;
    for (int i = 0; ok && i < (xt_kept ? 1 : n_iter); ++i) {
      for (int c = 0; c < my_boxes * subs; ++c) {
        if (!mbar_wait_warp(smem_u32(&sh.xe[xs]), xph, &sh.ctl, p.status, 830)) { ok = false; break; }
        if (elect_one()) {
          const uint32_t bar = smem_u32(&sh.xf[xs]), dst = smem_u32(smem_xt + xs * xt_stage);
          mbar_arrive_expect_tx(bar, (uint32_t)xt_stage);
          const int f = subs == 1 ? (box0 + c) * 128 : (box0 + (c >> 1)) * 128 + p.uw * (c & 1);      // the other team's features are 64 further
          for (int kb = 0; kb < nkb; ++kb) {
            tma_load_2d(dst + kb * p.uw * 256, &map_xt, bar, kb * 64, f);
            tma_load_2d(dst + kb * p.uw * 256 + p.uw * 128, &map_xt, bar, kb * 64, f + 64);
          }
        }
        __syncwarp();
        if (++xs == xt_ring) { xs = 0; xph ^= 1u; }
      }
    }
  } else if (warp == 3) {
    // ------------------------------ stores of updated boxes ------------------------------
    uint32_t ws = 0, wph = 0;
    bool ok = true;
    for (int i = 0; ok && i < n_iter; ++i) {
      int ci, row0;
      tile_at(i, ci, row0);
      const CUtensorMap* wm = p.w_maps + ci;
      for (int bx = 0; bx < my_boxes; ++bx) {
        if (!mbar_wait_warp(smem_u32(&sh.wd[ws]), wph, &sh.ctl, p.status, 841)) { ok = false; break; }
        if (lane == 0) {
          tma_store_2d(wm, smem_u32(smem_w + ws * kWSlot), (box0 + bx) * 128, row0);
          if (!W8 && (box0 + bx) * 128 + 64 < d) tma_store_2d(wm, smem_u32(smem_w + ws * kWSlot + kSlBox), (box0 + bx) * 128 + 64, row0);
          bulk_commit_group();
          bulk_wait_read_all();
          mbar_arrive(smem_u32(&sh.we[ws]));
        }
        __syncwarp();
        if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
      }
    }
    if (lane == 0) bulk_wait_all();
    __syncwarp();
  } else if (warp < 4 + kSlGWarps) {
    // ------------------------------ G ------------------------------
    warp_regs<kSlLaunchRegs, slim_g_regs(KAHAN != kKahanNone && !LOSS)>();
    const int q = warp & 3;                                      // TMEM lane quarter
    const int row = q * 32 + lane;                               // label row within the tile
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const uint32_t mrow = smem_u32(smem_m + (warp - 4) * 64);
    const uint32_t smem_g_peer = mapa_shared(smem_u32(smem_g), rank ^ 1u);
    const uint32_t ready_peer = mapa_shared(smem_u32(&sh.g_ready[0]), rank ^ 1u);
    const int h = (warp - 4) >> 2;                               // every other sixteen (or eight) batch columns
    const int b0 = (int)rank * nz;                               // this CTA's half of the batch
    double loss = 0.0;                                           // over all tiles of the cluster
    uint32_t zb = 0, zph = 0, gb = 0, gph = 1u;
    // the positives' range of a tile is read while the one before is at work
    auto bucket = [&](int i, int& beg, int& end) {
      int ci, row0;
      tile_at(i, ci, row0);
      const int bkt = ci * p.bkt_per_chunk + (row0 >> 7);
      beg = p.bucket_off[bkt];
      end = p.bucket_off[bkt + 1];
    };
    if constexpr (SPLIT) {                                       // (every warp the same)
      if (2 * lane < nz) *reinterpret_cast<float2*>(sh.x_scale + 2 * lane) = *reinterpret_cast<const float2*>(p.x_scale + b0 + 2 * lane);
      __syncwarp();
    }
    int next_beg, next_end;
    bucket(0, next_beg, next_end);
    for (int i = 0; i < n_iter; ++i) {
      int ci, row0;
      tile_at(i, ci, row0);
      const bool row_valid = row0 + row < (ci == p.n_chunks - 1 ? p.rows_last : p.rows_full);
      // positives of this row, a bit for each batch column (a duplicate pair counts once)
      uint2 bits = make_uint2(0u, 0u);
      if (next_end > next_beg) bits = slim_positives(p.bucket_ent, next_beg, next_end, q, b0, nz, mrow);
      if (i + 1 < n_iter) bucket(i + 1, next_beg, next_end);
      if (!mbar_wait_warp(smem_u32(&sh.z_full[zb]), zph, &sh.ctl, p.status, 850) ||
          !mbar_wait_warp(smem_u32(&sh.g_empty[gb]), gph, &sh.ctl, p.status, 851))
        break;
      tc_fence_after();
      // the other half comes from the peer
      if (warp == 4 && lane == 0) mbar_expect_tx(smem_u32(&sh.g_ready[gb]), (uint32_t)(128 * nz * 2));
      const uint32_t z_at = tmem_base + lane_sel + z_col + zb * (uint32_t)nz;
      SoftplusSum sp;
      float minus = 0.f;
      // eight batch columns, from c on
      auto piece = [&](int c, const uint32_t (&v)[8]) {
        const int b = b0 + c;
        uint32_t zz[4], out[4];
        [[maybe_unused]] uint64_t sc[2] = {0ull, 0ull};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (SPLIT && (e & 1) == 0) shared_scales(smem_u32(sh.x_scale) + 4u * (uint32_t)(c + 2 * e), sc);
          zz[e] = SPLIT ? scaled_bf16x2(v[2 * e], v[2 * e + 1], sc[e & 1])
                        : pack_bf16x2(__uint_as_float(v[2 * e]) * p.w_scale, __uint_as_float(v[2 * e + 1]) * p.w_scale);
          const float z0 = __uint_as_float(zz[e] << 16), z1 = __uint_as_float(zz[e] & 0xFFFF0000u);
          out[e] = pack_bf16x2(fast_sigmoid(z0), fast_sigmoid(z1));
          if (LOSS) {
            const int left = p.batch - (b + 2 * e);      // the same for the whole warp
            if (left > 1) sp.add(z0, z1);
            else if (left == 1) sp.add(z0);
          }
        }
        const uint32_t pos8 = ((c & 32 ? bits.y : bits.x) >> (c & 31)) & 0xFFu;
        if (pos8 != 0u) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t pos = (pos8 >> (2 * e)) & 3u;       // bf16(sigmoid) - 1 in bf16 arithmetic
            float lo = __uint_as_float(out[e] << 16), hi = __uint_as_float(out[e] & 0xFFFF0000u);
            if (pos & 1u) lo = bf16_round(lo - 1.0f);
            if (pos & 2u) hi = bf16_round(hi - 1.0f);
            out[e] = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
            if (LOSS) minus += ((pos & 1u) ? __uint_as_float(zz[e] << 16) : 0.f) + ((pos & 2u) ? __uint_as_float(zz[e] & 0xFFFF0000u) : 0.f);
          }
        }
        // rows beyond the chunk and batch columns beyond the batch carry G = 0
        if (!row_valid) out[0] = out[1] = out[2] = out[3] = 0u;
        else if (b + 8 > p.batch) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (b + 2 * e >= p.batch) out[e] = 0u;
            else if (b + 2 * e + 1 >= p.batch) out[e] &= 0xFFFFu;
          }
        }
        const uint32_t at = (gb * (uint32_t)nkb + (uint32_t)(b >> 6)) * kSlBox + (uint32_t)(row * 128) + ((((uint32_t)(b & 63) >> 3) ^ (uint32_t)(row & 7)) << 4);
        *reinterpret_cast<uint4*>(smem_g + at) = make_uint4(out[0], out[1], out[2], out[3]);
        st_async_16(smem_g_peer + at, out, ready_peer + 8u * gb);
      };
      uint32_t va[8], vb[8];
      if (!W8 && LOSS) {
        // The last sixteen columns of 16, and in rows of three boxes and more of 48, by both halves of the warps: 300 000 x 384 at batch 96 240 ->
        // 229 us, 250 000 x 512 221 -> 210, but 400 000 x 256 200 -> 207.  (e4m3 weights lose by it, 400 000 x 256 147 and 161: the workers want the
        // issue slots.)
        const int whole = p.n_boxes > 2 || nz == 16 ? nz & ~31 : nz;
#pragma unroll 1
        for (int c16 = 16 * h; c16 < whole; c16 += 32) {
          tmem_ld8(z_at + (uint32_t)c16, va);
          tmem_ld8(z_at + (uint32_t)c16 + 8u, vb);
          tmem_ld_wait_for(va, vb);
          piece(c16, va);
          piece(c16 + 8, vb);
        }
        if (whole != nz) {
          tmem_ld8(z_at + (uint32_t)(whole + 8 * h), va);
          tmem_ld_wait_for(va);
          piece(whole + 8 * h, va);
        }
      } else if (nz == 16) {                                     // all eight warps at work
        tmem_ld8(z_at + 8u * (uint32_t)h, va);
        tmem_ld_wait_for(va);
        piece(8 * h, va);
      } else {
#pragma unroll 1
        for (int c16 = 16 * h; c16 < nz; c16 += 32) {
          tmem_ld8(z_at + (uint32_t)c16, va);
          tmem_ld8(z_at + (uint32_t)c16 + 8u, vb);
          tmem_ld_wait_for(va, vb);
          piece(c16, va);
          piece(c16 + 8, vb);
        }
      }
      tc_fence_before();
      if (LOSS && row_valid) loss += (double)(sp.value() - minus);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&sh.z_empty[zb]));
        mbar_arrive(smem_u32(&sh.g_ready[gb]));
      }
      if (++zb == (uint32_t)p.z_bufs) { zb = 0; zph ^= 1u; }
      if (++gb == (uint32_t)p.g_bufs) { gb = 0; gph ^= 1u; }
    }
    if (LOSS) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
      if (lane == 0 && p.loss_partial != nullptr) p.loss_partial[blockIdx.x * kSlGWarps + (warp - 4)] = loss;
    }
  } else {
    // ------------------------------ workers ------------------------------
    warp_regs<kSlLaunchRegs, slim_worker_regs(KAHAN != kKahanNone && !LOSS)>();
    const int wk = warp - 4 - kSlGWarps, q = warp & 3, hw = wk >> 2;         // q: TMEM lane quarter
    const uint32_t team = (uint32_t)hw & 1u;
    const int hh = hw >> 1;
    const int row = q * 32 + lane;                               // label row within the tile
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    uint32_t ws = 0, wph = 0, ss = 0, sph = 1u, ub = 0, uph = 0;
    bool ok = true;
    // gx of box bx: out of TMEM into the cluster's slot of `partial`.  Features are lanes, batch rows columns: four lanes
    // exchange theirs, then each has four neighbouring features of a row and a warp whole 128-byte lines.  An
    // element is always handled by the same thread: its additions stay in order.
    auto drain_gx = [&](int bx, bool add) {
      const int f = (box0 + bx) * 128 + (row & ~3), gspan = nb >> 2;
      for (int c8 = 0; c8 < gspan; c8 += 8) {
        const int b0 = hw * gspan + c8;
        uint32_t v[8];
        tmem_ld8(tmem_base + lane_sel + (uint32_t)(bx * nb + b0), v);
        tmem_ld_wait_for(v);
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
          transpose4(v + h, lane);
          const int b = b0 + h + (lane & 3);
          if (b < p.batch && f < d) {
            float* dst = p.partial + ((size_t)worker * nb + b) * d + f;
            if (add) {
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(__uint_as_float(v[h])),
                           "f"(__uint_as_float(v[h + 1])), "f"(__uint_as_float(v[h + 2])), "f"(__uint_as_float(v[h + 3]))
                           : "memory");
            } else {
              *reinterpret_cast<uint4*>(dst) = make_uint4(v[h], v[h + 1], v[h + 2], v[h + 3]);
            }
          }
        }
        __syncwarp();
      }
    };
    // What a thread reads and writes of a box sits at the same places of every box; the second of its two runs
    // of 16 features is one bit of the address away.
    const int ct0 = subs == 1 ? 32 * hh : 16 * hh;               // first column within the team's 64 features
    const uint32_t w_at0 = (uint32_t)(row * 128 + (((4 * (int)team + (ct0 >> 4)) ^ (row & 7)) << 4));
    const uint32_t s_at0 = (uint32_t)((int)team * kSlBox + row * 128 + (((ct0 >> 3) ^ (row & 7)) << 4));
    const uint32_t u_at0 = tmem_base + lane_sel + u_col + team * (uint32_t)p.uw + (uint32_t)ct0;
    const uint32_t w_flip = subs == 1 ? 16u : 32u, s_flip = subs == 1 ? 32u : 64u, q_step = subs == 1 ? 2u : 4u;
    const int f_first = box0 * 128 + 64 * (int)team + ct0;
    typename Upd::PhiloxRow pr;
    if (SR) Upd::philox_row(p.upd, (uint32_t)(p.upd.elem0 >> 35), pr);
    auto tiles = [&](int first, int end) {
      for (int i = first; ok && i < end; ++i) {
        int ci, row0;
        tile_at(i, ci, row0);
        const int crow = row0 + row;
        const unsigned long long erow =
            p.upd.elem0 + ((unsigned long long)ci * (unsigned long long)p.rows_full + (unsigned long long)crow) * (unsigned long long)d;
        const unsigned long long q0 = (erow + (unsigned long long)f_first) >> 3;
        if (SR && (uint32_t)(q0 >> 32) != pr.q_hi) Upd::philox_row(p.upd, (uint32_t)(q0 >> 32), pr);
        bool kahan_row = false, row_valid = false;
        if constexpr (KAHAN != kKahanNone) {
          kahan_row = ci == 0 && crow < p.upd.kahan_rows;
          row_valid = crow < (ci == p.n_chunks - 1 ? p.rows_last : p.rows_full);
        }
        for (int bx = 0; ok && bx < my_boxes; ++bx) {
          uint8_t* wbox = smem_w + ws * kWSlot;
          uint8_t* sbox = smem_s + ss * 2 * kSlBox;
          if (!W8 && ((i + 1) & p.gx_mask) == 0 && i + 1 < n_iter) {
            // a sum of gx ends with this tile
            if (!mbar_wait_warp(smem_u32(&sh.gf[ws]), wph, &sh.ctl, p.status, 857)) { ok = false; break; }
            tc_fence_after();
            drain_gx(bx, i > p.gx_mask);
          }
          uint32_t w_at = w_at0, s_at = s_at0, u_at = u_at0 + ub * 2u * (uint32_t)p.uw, ql = (uint32_t)q0 + 16u * (uint32_t)bx;
#pragma unroll 1
          for (int sb = 0; sb < 2; ++sb) {                         // 16 of the team's 64 features of the box at a time
            uint4 comp[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
            const int f0 = f_first + 128 * bx + (int)q_step * 8 * sb;       // (d is a multiple of 16: its sixteen are there or none of them)
            if (KAHAN != kKahanNone && kahan_row && row_valid && f0 < d)
              Upd::template kahan_fetch<KAHAN == kKahanE5m2>(p.upd, (size_t)crow * d + f0, comp);
            if (sb == 0 || subs == 2) {
              if (!mbar_wait_warp(smem_u32(&sh.uf[ub]), uph, &sh.ctl, p.status, 854)) { ok = false; break; }
              if (sb == 0) {
                if constexpr (U_WAITS) {
                  mbar_test_wait(smem_u32(&sh.wf[ws]), wph);       // landed before U was issued: acquires it
                } else if (!mbar_wait_warp(smem_u32(&sh.wf[ws]), wph, &sh.ctl, p.status, 858) ||
                           (!kLateWait && !mbar_wait_warp(smem_u32(&sh.se[ss]), sph, &sh.ctl, p.status, 859))) {
                  ok = false;
                  break;
                }
              }
              tc_fence_after();
            }
            uint32_t va[8], vb[8];
            tmem_ld8(u_at, va);
            tmem_ld8(u_at + 8u, vb);
            // bf16 weights lie where the copy of e4m3 ones goes
            uint4* wslot = reinterpret_cast<uint4*>(wbox + (W8 ? w_at : s_at));
            const uint4 w = *wslot;
            uint4* wslot_b = reinterpret_cast<uint4*>(wbox + (s_at ^ 16u));
            uint4 w_b = w;
            if constexpr (!W8) w_b = *wslot_b;
            uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
            if (SR) {
              if (ql < (uint32_t)q0 && pr.q_hi == (uint32_t)(q0 >> 32)) Upd::philox_row(p.upd, (uint32_t)(q0 >> 32) + 1u, pr);
              ra = Upd::philox(p.upd, pr, ql);
              rb = Upd::philox(p.upd, pr, ql + 1u);
            }
            tmem_ld_wait_for(va, vb);
            if (sb == 1 || subs == 2) {                            // the chunk is in registers: its columns are free
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&sh.ue[ub]));
              if (++ub == (uint32_t)p.u_bufs) { ub = 0; uph ^= 1u; }
            }
            // before anything is written: the buffer of the copy is free, the old bf16 weights have been multiplied
            auto may_write = [&]() {
              return U_WAITS || !kLateWait || sb != 0 || mbar_wait_warp(smem_u32(W8 ? &sh.se[ss] : &sh.gf[ws]), W8 ? sph : wph, &sh.ctl, p.status, 859);
            };
            if constexpr (W8) {
              uint32_t old[8];
              uint4 nw = w;
              if (KAHAN != kKahanNone && kahan_row) {
                if (row_valid && f0 < d) nw = Upd::template kahan16<KAHAN == kKahanE5m2>(p.upd, va, vb, w, ra, rb, (size_t)crow * d + f0, comp);
                e4m3x4_to_bf16x4(w.x, old[0], old[1]);
                e4m3x4_to_bf16x4(w.y, old[2], old[3]);
                e4m3x4_to_bf16x4(w.z, old[4], old[5]);
                e4m3x4_to_bf16x4(w.w, old[6], old[7]);
              } else {
                nw = Upd::update16(p.upd, va, vb, w, ra, rb, old);
              }
              if constexpr (!U_WAITS && kLateWait) __syncwarp();
              if (!may_write()) { ok = false; break; }
              *wslot = nw;
              // the old weights as bf16, where the tensor core reads them with the label row as contraction index
              *reinterpret_cast<uint4*>(sbox + s_at) = make_uint4(old[0], old[1], old[2], old[3]);
              *reinterpret_cast<uint4*>(sbox + (s_at ^ 16u)) = make_uint4(old[4], old[5], old[6], old[7]);
            } else {
              const uint4 nw = make_uint4(Upd::update2_bf16(p.upd, va[0], va[1], w.x, ra.x), Upd::update2_bf16(p.upd, va[2], va[3], w.y, ra.y),
                                          Upd::update2_bf16(p.upd, va[4], va[5], w.z, ra.z), Upd::update2_bf16(p.upd, va[6], va[7], w.w, ra.w));
              const uint4 nw_b = make_uint4(Upd::update2_bf16(p.upd, vb[0], vb[1], w_b.x, rb.x), Upd::update2_bf16(p.upd, vb[2], vb[3], w_b.y, rb.y),
                                            Upd::update2_bf16(p.upd, vb[4], vb[5], w_b.z, rb.z), Upd::update2_bf16(p.upd, vb[6], vb[7], w_b.w, rb.w));
              if (!may_write()) { ok = false; break; }
              *wslot = nw;
              *wslot_b = nw_b;
            }
            w_at ^= w_flip;
            s_at ^= s_flip;
            u_at = subs == 1 ? u_at + 16u : u_at0 + ub * 2u * (uint32_t)p.uw;
            ql += q_step;
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh.wd[ws]));
          if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
          if (++ss == (uint32_t)p.s_bufs) { ss = 0; sph ^= 1u; }
        }
      }
    };
    if constexpr (BOUND) {
      uint32_t gxph = 0;
      for (int i = 0; ok && i < n_iter; i += p.gx_tiles, gxph ^= 1u) {
        tiles(i, min(n_iter, i + p.gx_tiles));
        if (!ok || my_boxes == 0) continue;
        ok = mbar_wait_warp(smem_u32(&sh.gx_full), gxph, &sh.ctl, p.status, 855);
        tc_fence_after();
        for (int bx = 0; ok && bx < my_boxes; ++bx) drain_gx(bx, i > 0);
        tc_fence_before();
      }
    } else {
      tiles(0, n_iter);
      if (ok && my_boxes > 0 && mbar_wait_warp(smem_u32(&sh.gx_full), 0u, &sh.ctl, p.status, 855)) {
        tc_fence_after();
        for (int bx = 0; bx < my_boxes; ++bx) drain_gx(bx, !W8 && n_iter > p.gx_mask + 1);
      }
    }
  }

  __syncwarp();
  if (sh.ctl.abort) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  cluster_sync_all();                     // the peer may still be writing to this CTA's shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace xmc
