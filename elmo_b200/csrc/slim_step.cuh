// The whole layer step for small batches (bf16 weights, or e4m3 with real-FP8 arithmetic) in ONE kernel: forward, loss
// gradient, grad_X and the fused weight update of a label tile while its weights are on the chip.
//
// With the three separate kernels (forward, grad_X, update) every weight is fetched three times by kernels that
// each ramp up and drain once per weight chunk; at batches up to 128 the contractions are so thin that this,
// not arithmetic, is what a step consists of.  Here a cluster of two CTAs takes tiles of 128 label rows and
// shares a tile twice over: by BATCH for the logits (each CTA multiplies the whole weight rows with its half of
// the batch and sends its half of G to the other through distributed shared memory), by FEATURES for the rest
// (each CTA updates, and accumulates grad_X for, its half of the 128-feature boxes).
//
// This kernel, 670 091 x 768 e4m3: batch 32 451 us, 64 and 96 477 and 561, 128 645.  (When it was made it took 492, 497, 588 and 655
// where the three kernels of the time took 660, 655, 738 and 761.)
// What bounds it is the stochastic-rounding arithmetic of the update (xmc_policies.cuh: 16 cycles per e4m3 weight
// and scheduler; the rest is arranged to hide behind it).  bf16, 300 000 x 768, batch 32: 415 and 259 us (at 128: 425
// and 413; 954 846 x 512 at 50: 919 and 573; 131 072 x 768 at 128: 213 and 195), of which the memory needs 141; what bounds it
// there is the chain of a tile, logits -> G -> the other CTA -> U -> update, and emptying the sums of gx (242 us without).  The dispatch goes up to batch 128 because
// the grad_X accumulators of half the features, half a Z and the update's chunks then just fit into the 512 columns
// of TMEM.
//
// bf16 weights need no copy for the tensor core: gx is multiplied from the box itself, together with the box's U and
// so before the workers, who wait for both, rewrite it in place.
//
//   warp 0       Z[128 labels x nb/2] += W box . X box (K = 128 e4m3 or 64 bf16 features a box): tcgen05.mma, and the
//                loads (128 rows x 128 bytes of weights and X, a small ring); asks L2 for the weights of the tile
//                after next.  bf16, twice the boxes: warp 20 does the loads (250 instead of 282 us at batch 32)
//   warp 1       issues the other tcgen05.mma:
//                  U[128 labels x 2 uw]     = G . X^T chunk            (bf16, K = batch)
//                  gx[128 features x nb]   += (old W box)^T . G        (bf16, K = 128 labels)
//                gx of all the CTA's boxes stays in TMEM until the last tile; with bf16 weights the workers add it to the
//                partial sums in memory every few tiles and it starts from zero (gx_mask; a long sum in the
//                accumulator loses digits).  (One warp for Z as well was the
//                kernel's critical path: its few hundred instructions a tile wait for their turn among the
//                workers' -- 13 000 cycles a tile however little the workers had to do.)
//   warp 2       loads for the update: the CTA's weight boxes once more (from L2) and X^T chunks
//   warp 3       stores updated boxes back
//   warps 4..19  logits -> sigmoid - y -> G (bf16, both CTAs' shared memory), a tile ahead of the update, a few of
//                the warps in turn (16 batch columns each); update
//                of the boxes in place, in two teams of eight warps that take one half of every box each and
//                drift apart, so that one computes while the other waits; the old weights, in registers
//                at that point, are written out as bf16 for the gx contraction on the way
//
// No updated box can be stored before BOTH CTAs have multiplied the old weights into Z: U needs all of G.
//
// TMEM columns: boxes0 x nb for gx, z_bufs x nb / 2 for Z, u_bufs x 2 uw for U.
#pragma once
#include "gemm_engine.cuh"
#include "numerics.cuh"
#include "xmc_policies.cuh"

namespace xmc {

constexpr int kSlWorkers = 16;
// bf16 weights: one warp more, for Z's loads (e4m3: it would leave 80 registers a thread, the update wants 96)
constexpr int slim_threads(bool w8) { return 128 + 32 * kSlWorkers + (w8 ? 0 : 32); }
constexpr int kSlBox = 128 * 128;               // one weight box: 128 rows x 128 bytes (features)
constexpr int kSlStaging = 2;
constexpr int kSlMaxZ = 4, kSlMaxW = 3, kSlMaxXt = 2, kSlG = 2;

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
  int gx_mask;                     // bf16: tiles that a grad_X accumulator sums up before it is added to `partial`, a power of two, minus one
  float w_scale;
  const int* bucket_off;
  const uint32_t* bucket_ent;
  double* loss_partial;            // [gridDim.x * kSlWorkers] or nullptr
  float* partial;                  // [clusters][nb][d]
  UpdParams upd;                   // kahan rows, learning rate, random stream; elem0 = element index of row 0 of chunk 0
  int* status;
};

struct SlimShared {
  uint64_t zf[kSlMaxZ], ze[kSlMaxZ];      // Z ring
  uint64_t z_full[2], z_empty[2];
  uint64_t g_ready[kSlG], g_empty[kSlG];        // G: own warps and the peer's bytes / the MMAs of both CTAs have read it
  uint64_t xf[kSlMaxXt], xe[kSlMaxXt];          // X^T chunks
  uint64_t wf[kSlMaxW], wd[kSlMaxW], we[kSlMaxW];   // weight boxes: landed, rewritten (and copied), stored
  uint64_t uf[2], ue[2];                        // update chunks
  uint64_t se[kSlStaging];                      // the copy of the old weights has been multiplied
  uint64_t gx_full;
  uint32_t tmem_base;
  Ctl ctl;
};

__host__ __device__ constexpr int slim_k_blocks(int nb) { return (nb + 63) / 64; }
__host__ __device__ constexpr int slim_smem_bytes(bool w8, int nb, int uw, int z_stages, int w_slots, int xt_stages) {
  return z_stages * (kSlBox + nb * 64) + w_slots * (w8 ? kSlBox : 2 * kSlBox) + (w8 ? kSlStaging * 2 * kSlBox : 0) + kSlG * slim_k_blocks(nb) * kSlBox +
         xt_stages * slim_k_blocks(nb) * uw * 256 + kSlWorkers * 128 + (int)sizeof(SlimShared);
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

// Positives of a bucket among the label rows 32 q + [0, 32) and the batch columns bw + [0, 16): lane i gets the columns of row
// 32 q + i; mrow: the warp's 32 words of shared memory.  A function that is called: of thousands of tiles a few dozen have
// positives, and the walk, inlined, cost every tile that has none.  One entry a turn, four inlined, this, us: e4m3
// 1 000 000 x 128 at batch 32 298, 313, 293; 600 000 x 768 at 128 596, 595, 583; bf16 700 000 x 320 at 8 356, 382, 345, 900 000 x
// 256 at 128 490, 505, 487.  Four entries a lane are under way at a time, without a branch for each: with one entry a turn the popular
// labels of 6 000 x 768 at batch 128, 20 positives a row, were 31 -> 39 us.  (Called once ahead of time, to have its instructions
// there, every kernel was 2 to 8 % slower.)
__device__ __noinline__ uint32_t slim_positives(const uint32_t* __restrict__ ents, int beg, int end, int q, int bw, uint32_t mrow) {
  const int lane = threadIdx.x & 31;
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(mrow + 4u * (uint32_t)lane), "r"(0u) : "memory");
  __syncwarp();
  for (int e0 = beg + lane; e0 < end; e0 += 128) {
    uint32_t ent[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) ent[u] = e0 + 32 * u < end ? ents[e0 + 32 * u] : 0xFFFFFFFFu;   // no row of any tile
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t lrow = ent[u] >> 16, c = (ent[u] & 0xFFFFu) - (uint32_t)bw;
      const uint32_t in = (uint32_t)((lrow >> 5) == (uint32_t)q) & (uint32_t)(c < 16u);
      asm volatile("{.reg .pred p; setp.ne.u32 p, %2, 0; @p red.shared.or.b32 [%0], %1;}" ::"r"(mrow + 4u * (lrow & 31u)),
                   "r"(1u << (c & 31u)), "r"(in) : "memory");
    }
  }
  __syncwarp();
  uint32_t bits;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(bits) : "r"(mrow + 4u * (uint32_t)lane) : "memory");
  return bits;
}

// What compensates the first rows of chunk 0.  A kernel for either type: with both in one, bf16 terms took 1 to 4 % longer.
enum KahanTerms { kKahanNone, kKahanBf16, kKahanE5m2 };

// AHEAD2: U runs two boxes ahead of gx, which waits for the workers, instead of one; it is there then when the workers
// come to the box.  (A tile's G is made one box before its end, so two boxes are the most; a CTA with a single box a tile
// stays at one, its next G would wait for the gx behind it.)  What U's first chunk told the workers with one, that the weights
// have landed and the staging buffer is free, they wait for themselves: a kernel of its own, as those waits cost 2 % where
// they are not needed.  The host's rule says where it pays.
template <bool W8, bool SR, bool LOSS, KahanTerms KAHAN, bool AHEAD2 = false>
__global__ void __launch_bounds__(slim_threads(W8), 1)
slim_step_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_xt,
                 const __grid_constant__ SlimParams p) {
  using Upd = UpdPolicy<W8, SR, !W8, false, KAHAN != kKahanNone>;
  constexpr int kWSlot = W8 ? kSlBox : 2 * kSlBox;               // 128 features of 128 rows
  constexpr int kZFeatures = W8 ? 128 : 64;                      // features of a Z box: 128 bytes of a row
  extern __shared__ __align__(1024) uint8_t smem[];
  const int nb = p.nb, nz = nb >> 1, nkb = slim_k_blocks(nb), d = p.upd.d;
  const int z_stage = kSlBox + nz * 128, xt_stage = nkb * p.uw * 256;
  uint8_t* smem_z = smem;                                        // [stage][W box | X box]
  uint8_t* smem_w = smem_z + p.z_stages * z_stage;               // [slot][128 rows][128 B], bf16: two blocks of 64 features
  uint8_t* smem_s = smem_w + p.w_slots * kWSlot;                 // e4m3: [buffer][2 blocks of 64 features][128 rows][128 B]
  uint8_t* smem_g = smem_s + (W8 ? kSlStaging * 2 * kSlBox : 0);            // [buffer][blocks of 64 batch rows][128 labels][128 B]
  uint8_t* smem_xt = smem_g + kSlG * nkb * kSlBox;               // [stage][blocks of 64 batch rows][2 uw features][128 B]
  uint32_t* smem_m = reinterpret_cast<uint32_t*>(smem_xt + p.xt_stages * xt_stage);    // [worker][32 rows]
  SlimShared& sh = *reinterpret_cast<SlimShared*>(smem_m + kSlWorkers * 32);
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
      // 4 warps for every 16 batch columns, or all (see make_g)
      mbar_init(smem_u32(&sh.z_empty[i]), my_boxes > 1 ? (uint32_t)nz >> 2 : (uint32_t)kSlWorkers);
    }
    for (int i = 0; i < kSlG; ++i) { mbar_init(smem_u32(&sh.g_ready[i]), (uint32_t)nz >> 2); mbar_init(smem_u32(&sh.g_empty[i]), 2); }
    for (int i = 0; i < kSlMaxXt; ++i) { mbar_init(smem_u32(&sh.xf[i]), 1); mbar_init(smem_u32(&sh.xe[i]), 1); }
    for (int i = 0; i < kSlMaxW; ++i) {
      mbar_init(smem_u32(&sh.wf[i]), 1);
      mbar_init(smem_u32(&sh.wd[i]), kSlWorkers);
      mbar_init(smem_u32(&sh.we[i]), 1);
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
  if (warp == 0 || warp == 2 || warp == 3 || (!W8 && warp == 4 + kSlWorkers)) tensormap_acquire(p.w_maps, 0, p.n_chunks - 1);
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

  if (warp == 0 || (!W8 && warp == 4 + kSlWorkers)) {
    // ------------------------------ Z: loads and MMAs ------------------------------
    const uint32_t z0 = smem_u32(smem_z), zf0 = smem_u32(&sh.zf[0]), ze0 = smem_u32(&sh.ze[0]);
    const uint32_t stages = (uint32_t)p.z_stages;
    const int n_zboxes = (d + kZFeatures - 1) / kZFeatures;
    uint32_t ls = 0, lph = 1u;                                   // loading side: stage, parity of its release
    int li = 0, lk = 0, lci, lrow0;
    bool ok = true;
    tile_at(0, lci, lrow0);
    auto load = [&]() {                                          // the next box, once its stage is free
      if (li >= n_iter) return;
      if (lk == 0 && li + 2 < n_iter) {
        // the CTAs of a cluster fetch the same boxes: each asks L2 for every other one
        int cn, rn;
        tile_at(li + 2, cn, rn);
        if (elect_one())
          for (int k = (int)rank; k < n_zboxes; k += 2) tma_prefetch_2d(p.w_maps + cn, k * kZFeatures, rn);
        __syncwarp();
      }
      if (!mbar_wait_warp(ze0 + 8u * ls, lph, &sh.ctl, p.status, 800)) { ok = false; return; }
      if (elect_one()) {
        const CUtensorMap* wm = p.w_maps + lci;
        const uint32_t bar = zf0 + 8u * ls, dst = z0 + ls * (uint32_t)z_stage;
        mbar_arrive_expect_tx(bar, (uint32_t)z_stage);
        tma_load_2d(dst, wm, bar, lk * kZFeatures, lrow0);
        tma_load_2d(dst + kSlBox, &map_x, bar, lk * kZFeatures, (int)rank * nz);
      }
      __syncwarp();
      if (++ls == stages) { ls = 0; lph ^= 1u; }
      if (++lk == n_zboxes) {
        lk = 0;
        if (++li < n_iter) tile_at(li, lci, lrow0);
      }
    };
    if (warp != 0) {
      while (ok && li < n_iter) load();
    } else {
      constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
      constexpr uint32_t kFmt = W8 ? 0u : 1u;                    // e4m3, bf16
      const uint32_t idesc = make_idesc(128, (uint32_t)nz, kFmt, kFmt, 0u, 0u);
      if (W8)
        for (uint32_t i = 0; ok && i + 1 < stages; ++i) load();
      uint32_t s = 0, ph = 0, zb = 0, zph = 1u;
      for (int i = 0; ok && i < n_iter; ++i) {
        if (!mbar_wait_warp(smem_u32(&sh.z_empty[zb]), zph, &sh.ctl, p.status, 801)) break;
        const uint32_t d_tmem = tmem_base + z_col + zb * (uint32_t)nz;
        for (int k = 0; k < n_zboxes; ++k) {
          if (W8) load();
          if (!ok || !mbar_wait_warp(zf0 + 8u * s, ph, &sh.ctl, p.status, 802)) { ok = false; break; }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t a = smem_desc_lo(z0 + s * (uint32_t)z_stage, 16), b = a + (kSlBox >> 4);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
              if constexpr (W8) umma_f8_lohi(d_tmem, a + 2u * u, b + 2u * u, desc_hi, idesc, (k | (int)u) ? 1u : 0u);
              else umma_f16_lohi(d_tmem, a + 2u * u, b + 2u * u, desc_hi, idesc, (k | (int)u) ? 1u : 0u);
            }
            umma_commit(ze0 + 8u * s);
            if (k + 1 == n_zboxes) umma_commit(smem_u32(&sh.z_full[zb]));
          }
          __syncwarp();
          if (++s == stages) { s = 0; ph ^= 1u; }
        }
        if (++zb == (uint32_t)p.z_bufs) { zb = 0; zph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer for U and gx ------------------------------
    constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
    const uint32_t idesc_u = make_idesc(128, 2u * (uint32_t)p.uw, 1u, 1u, 0u, 0u);
    const uint32_t idesc_g = make_idesc(128, (uint32_t)nb, 1u, 1u, 1u, 1u);
    const uint32_t g_lo0 = smem_desc_lo(smem_u32(smem_g), 16), g_lo_mn0 = smem_desc_lo(smem_u32(smem_g), kSlBox);
    // the old weights for gx: the e4m3 boxes' copies, the bf16 boxes themselves
    const uint32_t xt_lo0 = smem_desc_lo(smem_u32(smem_xt), 16), s_lo0 = smem_desc_lo(smem_u32(W8 ? smem_s : smem_w), kSlBox);
    const uint32_t g_step = (uint32_t)(nkb * kSlBox) >> 4, xt_blk = (uint32_t)p.uw * 16u;
    uint32_t xs = 0, xph = 0, ub = 0, uph = 0;                   // X^T stage, U buffer
    uint32_t ws = 0, wph = 0, ss = 0, sph = 0;                   // weight slot and staging buffer of the next U's box
    uint32_t gs = 0, gph = 0, gss = 0;                           // ... and of the next gx's
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, int where) {
      if (ok && !mbar_wait_warp(smem_u32(bar), parity, &sh.ctl, p.status, where)) ok = false;
      return ok;
    };
    // gx of box bx of tile i from the old weights at descriptor a
    auto mma_gx = [&](int i, int bx, uint32_t a) {
      // both operands MN-major: blocks of 64 elements kSlBox apart, one MMA eats 16 label rows = 2048 B
      const uint32_t b = g_lo_mn0 + (uint32_t)(i & 1) * g_step, dt = tmem_base + (uint32_t)(bx * nb);
      umma_f16_lohi(dt, a, b, desc_hi, idesc_g, (W8 ? i : i & p.gx_mask) ? 1u : 0u);
#pragma unroll
      for (uint32_t u = 1; u < 8; ++u) umma_f16_lohi(dt, a + 128u * u, b + 128u * u, desc_hi, idesc_g, 1u);
    };
    // Update chunk c of box bx of tile i.  With the first one everything the workers need for the box is there, so they
    // wait for U alone: the weights have landed, and the staging buffer (bf16: the box itself) has been multiplied.
    // (Two boxes ahead that would hold U up: there the workers see to it.)
    auto issue_u = [&](int i, int bx, int c) {
      const uint32_t gb = (uint32_t)i & 1u;
      if (!wait(&sh.xf[xs], xph, 814) || !wait(&sh.ue[ub], uph ^ 1u, 815)) return;
      if (!AHEAD2 && c == 0 && (!wait(&sh.wf[ws], wph, 816) || (W8 && !wait(&sh.se[ss], sph ^ 1u, 817)))) return;
      // bf16: a new sum of gx begins with this chunk, so the old one has to be out of TMEM.  Its workers were at the
      // same box of the tile before: with two boxes and more U's buffers have shown that they are past it.
      if (!W8 && c == 0 && my_boxes == 1 && i > 0 && (i & p.gx_mask) == 0 && !wait(&sh.wd[gs], gph, 818)) return;
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
        if (!W8 && c == 0) mma_gx(i, bx, s_lo0 + ws * (2u * kSlBox >> 4));
        umma_commit(smem_u32(&sh.uf[ub]));
        umma_commit(smem_u32(&sh.xe[xs]));
      }
      __syncwarp();
      if (c == 0) {
        if (!W8 && i > 0 && ++gs == (uint32_t)p.w_slots) { gs = 0; gph ^= 1u; }
        if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
        if (++ss == kSlStaging) { ss = 0; sph ^= 1u; }
      }
      if (++xs == (uint32_t)p.xt_stages) { xs = 0; xph ^= 1u; }
      if (++ub == (uint32_t)p.u_bufs) { ub = 0; uph ^= 1u; }
    };
    // gx of a box of tile i, once its old e4m3 weights have been copied
    auto issue_gx = [&](int i, int bx) {
      if (!wait(&sh.wd[gs], gph, 812)) return;
      tc_fence_after();
      if (elect_one()) {
        mma_gx(i, bx, s_lo0 + gss * (2u * kSlBox >> 4));
        umma_commit(smem_u32(&sh.se[gss]));
      }
      __syncwarp();
      if (++gs == (uint32_t)p.w_slots) { gs = 0; gph ^= 1u; }
      gss ^= 1u;
    };
    auto g_there = [&](int i) {
      const uint32_t gb = (uint32_t)i & 1u;
      if (!wait(&sh.g_ready[gb], (uint32_t)(i >> 1) & 1u, 813)) return;
      mbar_acquire_cluster(smem_u32(&sh.g_ready[gb]), (uint32_t)(i >> 1) & 1u);
      fence_proxy_async();                          // the peer's half of G came by generic-proxy stores
    };
    const int mb = max(1, my_boxes), ahead = AHEAD2 && mb > 1 ? 2 : 1;
    g_there(0);
    if (my_boxes > 0)
      for (int k = 0; k < ahead; ++k)
        for (int c = 0; c < subs; ++c) issue_u(0, k, c);
    for (int i = 0; ok && i < n_iter; ++i) {
      for (int bx = 0; ok && bx < mb; ++bx) {
        const bool wrap = bx + ahead >= mb;
        const int in = wrap ? i + 1 : i, bn = bx + ahead - (wrap ? mb : 0);     // the box U comes to
        if (bn == 0 && in < n_iter) g_there(in);
        if (my_boxes > 0) {
          if (in < n_iter) issue_u(in, bn, 0);
          if constexpr (W8) issue_gx(i, bx);
          if (subs == 2 && in < n_iter) issue_u(in, bn, 1);
        }
      }
      // (not for the last two tiles: nobody waits for those buffers again, and a late arrival at the peer could meet
      // the shared memory of the next kernel there)
      if (i + 2 < n_iter && ok && elect_one()) umma_commit_both(smem_u32(&sh.g_empty[i & 1]));
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(smem_u32(&sh.gx_full));
    __syncwarp();
  } else if (warp == 2) {
    // ------------------------------ loads for the update ------------------------------
    uint32_t ws = 0, wph = 0, xs = 0, xph = 0;
    bool ok = true;
    for (int i = 0; ok && i < n_iter; ++i) {
      int ci, row0;
      tile_at(i, ci, row0);
      const CUtensorMap* wm = p.w_maps + ci;
      for (int bx = 0; ok && bx < my_boxes; ++bx) {
        auto load_w = [&]() {
          if (!mbar_wait_warp(smem_u32(&sh.we[ws]), wph ^ 1u, &sh.ctl, p.status, 820 + (int)ws)) { ok = false; return; }
          if (elect_one()) {
            const uint32_t bar = smem_u32(&sh.wf[ws]);
            mbar_arrive_expect_tx(bar, kWSlot);
            tma_load_2d(smem_u32(smem_w + ws * kWSlot), wm, bar, (box0 + bx) * 128, row0);
            if constexpr (!W8) tma_load_2d(smem_u32(smem_w + ws * kWSlot + kSlBox), wm, bar, (box0 + bx) * 128 + 64, row0);
          }
          __syncwarp();
          if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
        };
        // Where U runs two boxes ahead X^T goes first, as U does not wait for the weights: their slot is free only when
        // the workers have left it.
        if constexpr (!AHEAD2) load_w();
        for (int c = 0; ok && c < subs; ++c) {
          if (!mbar_wait_warp(smem_u32(&sh.xe[xs]), xph ^ 1u, &sh.ctl, p.status, 830 + (int)xs)) { ok = false; break; }
          if (elect_one()) {
            const uint32_t bar = smem_u32(&sh.xf[xs]), dst = smem_u32(smem_xt + xs * xt_stage);
            mbar_arrive_expect_tx(bar, (uint32_t)xt_stage);
            const int f = (box0 + bx) * 128 + p.uw * c;           // the other team's features are 64 further
            for (int kb = 0; kb < nkb; ++kb) {
              tma_load_2d(dst + kb * p.uw * 256, &map_xt, bar, kb * 64, f);
              tma_load_2d(dst + kb * p.uw * 256 + p.uw * 128, &map_xt, bar, kb * 64, f + 64);
            }
          }
          __syncwarp();
          if (++xs == (uint32_t)p.xt_stages) { xs = 0; xph ^= 1u; }
        }
        if constexpr (AHEAD2) {
          if (ok) load_w();
        }
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
  } else {
    // ------------------------------ workers ------------------------------
    const int wk = warp - 4, q = warp & 3, hw = wk >> 2;         // q: TMEM lane quarter
    const uint32_t team = (uint32_t)hw & 1u;
    const int hh = hw >> 1;
    const int row = q * 32 + lane;                               // label row within the tile
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    // duty for G: of the four warps of a quarter, nz / 16 a tile in turn
    const int n_duty = nz >> 4;
    const uint32_t mrow = smem_u32(smem_m + wk * 32);
    const uint32_t smem_g_peer = mapa_shared(smem_u32(smem_g), rank ^ 1u);
    const uint32_t ready_peer = mapa_shared(smem_u32(&sh.g_ready[0]), rank ^ 1u);
    float loss = 0.f;
    uint32_t ws = 0, wph = 0, ss = 0, ub = 0, uph = 0;
    [[maybe_unused]] uint32_t sph = 1u;                          // parity of the staging buffer's release
    bool ok = true;
    // Z of tile i -> G, 16 columns of this CTA's half of the batch
    auto make_g = [&](int i) {
      const int part = (hw + i * n_duty) & 3;
      const int zb = p.z_bufs == 2 ? i & 1 : 0;
      const uint32_t zph = (uint32_t)(p.z_bufs == 2 ? i >> 1 : i) & 1u;
      if (part >= n_duty) {
        // Not on duty.  A later wait for z_full must find the phase it waits for current or just completed.
        // With two boxes and more, this tile's U has shown the warp that the phase before is over; else the
        // warp waits along for every phase, and none can pass it by because z_empty counts it.
        if (my_boxes > 1) return true;
        if (!mbar_wait_warp(smem_u32(&sh.z_full[zb]), zph, &sh.ctl, p.status, 849)) return false;
        if (lane == 0) mbar_arrive(smem_u32(&sh.z_empty[zb]));
        __syncwarp();
        return true;
      }
      int ci, row0;
      tile_at(i, ci, row0);
      const bool row_valid = row0 + row < (ci == p.n_chunks - 1 ? p.rows_last : p.rows_full);
      const int bkt = ci * p.bkt_per_chunk + (row0 >> 7);
      const int bkt_beg = p.bucket_off[bkt], bkt_end = p.bucket_off[bkt + 1];
      const int bw = (int)rank * nz + 16 * part;
      // positives of this warp's rows and columns, one word per row (a duplicate pair counts once)
      uint32_t bits = 0u;
      if (bkt_end > bkt_beg) {
        bits = slim_positives(p.bucket_ent, bkt_beg, bkt_end, q, bw, mrow);
      }
      const int gb = i & 1;
      if (!mbar_wait_warp(smem_u32(&sh.z_full[zb]), zph, &sh.ctl, p.status, 850) ||
          !mbar_wait_warp(smem_u32(&sh.g_empty[gb]), (uint32_t)((i >> 1) & 1) ^ 1u, &sh.ctl, p.status, 851))
        return false;
      tc_fence_after();
      // the other half comes from the peer
      if (part == 0 && q == 0 && lane == 0) mbar_expect_tx(smem_u32(&sh.g_ready[gb]), (uint32_t)(128 * nz * 2));
      const uint32_t at0 = (uint32_t)((gb * nkb + (bw >> 6)) * kSlBox + row * 128), piece0 = (uint32_t)(bw & 63) >> 3;
      SoftplusSum sp;
#pragma unroll
      for (int c8 = 0; c8 < 16; c8 += 8) {
        uint32_t v[8], out[4];
        tmem_ld8(tmem_base + lane_sel + z_col + (uint32_t)(zb * nz + 16 * part + c8), v);
        tmem_ld_wait_for(v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t zz = pack_bf16x2(__uint_as_float(v[2 * e]) * p.w_scale, __uint_as_float(v[2 * e + 1]) * p.w_scale);
          const float z0 = __uint_as_float(zz << 16), z1 = __uint_as_float(zz & 0xFFFF0000u);
          uint32_t s2 = pack_bf16x2(fast_sigmoid(z0), fast_sigmoid(z1));
          if (bits != 0u) {
            const uint32_t pos = (bits >> (c8 + 2 * e)) & 3u;    // bf16(sigmoid) - 1 in bf16 arithmetic
            float lo = __uint_as_float(s2 << 16), hi = __uint_as_float(s2 & 0xFFFF0000u);
            if (pos & 1u) lo = bf16_round(lo - 1.0f);
            if (pos & 2u) hi = bf16_round(hi - 1.0f);
            s2 = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
            if (LOSS && row_valid) loss -= ((pos & 1u) ? z0 : 0.f) + ((pos & 2u) ? z1 : 0.f);
          }
          if (LOSS) {
            const int left = p.batch - (bw + c8 + 2 * e);         // the same for the whole warp
            if (left > 1) sp.add(z0, z1);
            else if (left == 1) sp.add(z0);
          }
          out[e] = s2;
        }
        // rows beyond the chunk and batch columns beyond the batch carry G = 0
        if (!row_valid) out[0] = out[1] = out[2] = out[3] = 0u;
        else if (bw + c8 + 8 > p.batch) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int b = bw + c8 + 2 * e;
            if (b >= p.batch) out[e] = 0u;
            else if (b + 1 >= p.batch) out[e] &= 0xFFFFu;
          }
        }
        const uint32_t at = at0 + (((piece0 + (uint32_t)(c8 >> 3)) ^ (uint32_t)(row & 7)) << 4);
        *reinterpret_cast<uint4*>(smem_g + at) = make_uint4(out[0], out[1], out[2], out[3]);
        st_async_16(smem_g_peer + at, out, ready_peer + 8u * (uint32_t)gb);
      }
      tc_fence_before();
      fence_proxy_async();
      if (LOSS && row_valid) loss += sp.value();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&sh.z_empty[zb]));
        mbar_arrive(smem_u32(&sh.g_ready[gb]));
      }
      return true;
    };
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
    // make_g stands in one place, inside the loop, or in two, before the loop and in it: which one is faster was measured for each
    // kind of kernel.  One / two, us: bf16 900 000 x 256 at batch 8 271 / 284, at 128 487 / 503; e4m3 with the loss 600 000 x 256 at
    // 6 230 / 242, 500 000 x 320 at 100 373 / 395; compensated rows to nearest 700 000 x 192 at 6 201 / 226, 300 000 x 768 at 100
    // 302 / 300.  Else two: e4m3 to nearest 600 000 x 256 at 128 265 / 244, compensated 500 000 x 768 at 64 493 / 485, and with the
    // loss 500 000 x 320 at 100 534 / 516.
    constexpr bool kOnePlace = !W8 || (KAHAN == kKahanNone ? LOSS : !SR);
    [[maybe_unused]] int g_next = 0;                             // the tile whose G comes next
    if constexpr (!kOnePlace) ok = make_g(0);
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
    for (int i = 0; ok && i < n_iter; ++i) {
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
      for (int bx = 0; ok && bx < max(1, my_boxes); ++bx) {
        // G of the next tile goes ahead of the tile's last box: the tensor core starts on it meanwhile
        if constexpr (!kOnePlace) {
          if (bx + 1 >= my_boxes && i + 1 < n_iter && !(ok = make_g(i + 1))) break;
        } else {
          for (const int upto = min(n_iter - 1, bx + 1 >= my_boxes ? i + 1 : i); ok && g_next <= upto; ++g_next) ok = make_g(g_next);
          if (!ok) break;
        }
        if (my_boxes == 0) break;
        uint8_t* wbox = smem_w + ws * kWSlot;
        uint8_t* sbox = smem_s + ss * 2 * kSlBox;
        if (!W8 && ((i + 1) & p.gx_mask) == 0 && i + 1 < n_iter) {
          // a sum of gx ends with this tile; the box's was multiplied together with its U
          if (!mbar_wait_warp(smem_u32(&sh.uf[ub]), uph, &sh.ctl, p.status, 857)) { ok = false; break; }
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
            if constexpr (AHEAD2) {
              if (sb == 0 && (!mbar_wait_warp(smem_u32(&sh.wf[ws]), wph, &sh.ctl, p.status, 858) ||
                              !mbar_wait_warp(smem_u32(&sh.se[ss]), sph, &sh.ctl, p.status, 859))) { ok = false; break; }
            } else {
              if (sb == 0) mbar_test_wait(smem_u32(&sh.wf[ws]), wph);      // landed before U was issued: acquires it
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
            *wslot = nw;
            // the old weights as bf16, where the tensor core reads them with the label row as contraction index
            *reinterpret_cast<uint4*>(sbox + s_at) = make_uint4(old[0], old[1], old[2], old[3]);
            *reinterpret_cast<uint4*>(sbox + (s_at ^ 16u)) = make_uint4(old[4], old[5], old[6], old[7]);
          } else {
            *wslot = make_uint4(Upd::update2_bf16(p.upd, va[0], va[1], w.x, ra.x), Upd::update2_bf16(p.upd, va[2], va[3], w.y, ra.y),
                                Upd::update2_bf16(p.upd, va[4], va[5], w.z, ra.z), Upd::update2_bf16(p.upd, va[6], va[7], w.w, ra.w));
            *wslot_b = make_uint4(Upd::update2_bf16(p.upd, vb[0], vb[1], w_b.x, rb.x), Upd::update2_bf16(p.upd, vb[2], vb[3], w_b.y, rb.y),
                                  Upd::update2_bf16(p.upd, vb[4], vb[5], w_b.z, rb.z), Upd::update2_bf16(p.upd, vb[6], vb[7], w_b.w, rb.w));
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
        ss ^= 1u;
        if (AHEAD2 && ss == 0) sph ^= 1u;
      }
    }
    if (ok && my_boxes > 0 && mbar_wait_warp(smem_u32(&sh.gx_full), 0u, &sh.ctl, p.status, 855)) {
      tc_fence_after();
      for (int bx = 0; bx < my_boxes; ++bx) drain_gx(bx, !W8 && n_iter > p.gx_mask + 1);
    }
    if (LOSS) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
      if (lane == 0 && p.loss_partial != nullptr) p.loss_partial[blockIdx.x * kSlWorkers + wk] = (double)loss;
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
