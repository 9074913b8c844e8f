// The whole layer step for small batches (e4m3 weights, real-FP8 arithmetic) in ONE kernel: forward, loss
// gradient, grad_X and the fused weight update of a label tile while its weights are on the chip.
//
// With the three separate kernels (forward, grad_X, update) every weight is fetched three times by kernels that
// each ramp up and drain once per weight chunk; at batches up to 128 the contractions are so thin that this,
// not arithmetic, is what a step consists of.  Here a cluster of two CTAs takes tiles of 128 label rows; the CTAs
// share a tile by FEATURES: each computes the tile's whole logits Z (the thin contraction: doing it twice
// costs less than exchanging halves) and then updates, and accumulates grad_X for, its own half of the
// 128-feature boxes.  What bounds it is the stochastic-rounding arithmetic of the update (xmc_policies.cuh:
// 16 cycles per weight and scheduler; the rest is arranged to hide behind it).
//
//   warp 0       loads for Z: the tile's weight boxes (128 rows x 128 bytes) and X, a ring of two stages
//   warp 1       issues every tcgen05.mma of the CTA:
//                  Z[128 labels x nb]      += W box . X box            (e4m3, K = 128 features a box)
//                  U[128 labels x uw]       = G . X^T chunk            (bf16, K = batch)
//                  gx[128 features x nb]   += (old W box)^T . G        (bf16, K = 128 labels)
//                gx of all the CTA's boxes stays in TMEM until the last tile
//   warp 2       loads for the update: the CTA's weight boxes once more (from L2) and X^T chunks
//   warp 3       stores updated boxes back
//   warps 4..19  per tile: logits -> sigmoid - y -> G (bf16, shared memory); then per chunk of uw features the
//                update in place; the old weights, in registers at that point, are written out as bf16
//                for the gx contraction on the way
//
// A tile's boxes may be stored only when BOTH CTAs have multiplied the old weights into Z: each CTA's
// workers signal the peer when their Z is complete and the store warp waits for that (a ring of 16 barriers:
// neither CTA can be more than 8 tiles ahead of the other, because un-stored boxes hold their slots).
//
// TMEM columns: boxes0 x nb for gx, nb for Z, 2 x uw for U.  Where that exceeds 512 (nb 128 at 768 features)
// U shares Z's columns, and Z of the next tile starts when this tile's update has been read out.
#pragma once
#include "gemm_engine.cuh"
#include "numerics.cuh"
#include "xmc_policies.cuh"

namespace xmc {

constexpr int kSlWorkers = 16;
constexpr int kSlThreads = 128 + 32 * kSlWorkers;
constexpr int kSlBox = 128 * 128;               // one weight box: 128 rows x 128 bytes (features)
constexpr int kSlZStages = 2, kSlXtStages = 2, kSlStaging = 2, kSlPeer = 16;
constexpr int kSlMaxW = 3, kSlMaxG = 2;

struct SlimParams {
  const CUtensorMap* w_maps;       // one per weight chunk: boxes of 128 rows x 128 bytes, 128-byte swizzle (device memory)
  int n_tiles;
  FastDiv div_tpc;                 // label tiles per chunk
  int rows_full, rows_last;        // label rows of every chunk but the last, of the last
  int n_chunks;
  int bkt_per_chunk;               // buckets (128 labels) per chunk
  int batch, nb;                   // batch rows; padded to a multiple of 32 (<= 128)
  int n_boxes;                     // 128-feature boxes of a row; CTA 0 of a cluster owns the first (n_boxes + 1) / 2
  int uw, alias;                   // features per update chunk (64 or 128); U shares Z's columns
  int w_slots, g_bufs;
  float w_scale;
  const int* bucket_off;
  const uint32_t* bucket_ent;
  double* loss_partial;            // [gridDim.x * kSlWorkers] or nullptr
  float* partial;                  // [clusters][nb][d]
  UpdParams upd;                   // kahan rows, learning rate, random stream; elem0 = element index of row 0 of chunk 0
  int* status;
};

struct SlimShared {
  uint64_t zf[kSlZStages], ze[kSlZStages];      // Z ring
  uint64_t z_full, z_empty;
  uint64_t g_ready, g_empty[kSlMaxG];
  uint64_t xf[kSlXtStages], xe[kSlXtStages];    // X^T chunks
  uint64_t wf[kSlMaxW], wd[kSlMaxW], we[kSlMaxW];   // weight boxes: landed, rewritten, stored
  uint64_t uf[2], ue[2];
  uint64_t sf[kSlStaging], se[kSlStaging];      // bf16 copies of the old weights
  uint64_t peer[kSlPeer];                       // the other CTA's Z of this tile is complete
  uint64_t gx_full;
  uint32_t tmem_base;
  Ctl ctl;
};

__host__ __device__ constexpr int slim_k_blocks(int nb) { return (nb + 63) / 64; }
__host__ __device__ constexpr int slim_smem_bytes(int nb, int uw, int w_slots, int g_bufs) {
  return kSlZStages * (kSlBox + nb * 128) + w_slots * kSlBox + kSlStaging * 2 * kSlBox + g_bufs * slim_k_blocks(nb) * kSlBox +
         kSlXtStages * slim_k_blocks(nb) * uw * 128 + kSlWorkers * 128 + (int)sizeof(SlimShared);
}

template <bool SR, bool LOSS, bool KAHAN>
__global__ void __launch_bounds__(kSlThreads, 1)
slim_step_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_xt,
                 const __grid_constant__ SlimParams p) {
  using Upd = UpdPolicy<true, SR, false, false, KAHAN>;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int nb = p.nb, nkb = slim_k_blocks(nb), d = p.upd.d;
  const int z_stage = kSlBox + nb * 128, xt_stage = nkb * p.uw * 128;
  uint8_t* smem_z = smem;                                        // [stage][W box | X box]
  uint8_t* smem_w = smem_z + kSlZStages * z_stage;               // [slot][128 rows][128 B]
  uint8_t* smem_s = smem_w + p.w_slots * kSlBox;                 // [buffer][2 blocks of 64 features][128 rows][128 B]
  uint8_t* smem_g = smem_s + kSlStaging * 2 * kSlBox;            // [buffer][blocks of 64 batch rows][128 labels][128 B]
  uint8_t* smem_xt = smem_g + p.g_bufs * nkb * kSlBox;           // [stage][blocks of 64 batch rows][uw features][128 B]
  uint32_t* smem_m = reinterpret_cast<uint32_t*>(smem_xt + kSlXtStages * xt_stage);    // [worker][32 rows]
  SlimShared& sh = *reinterpret_cast<SlimShared*>(smem_m + kSlWorkers * 32);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int worker = (int)(blockIdx.x >> 1), n_workers = (int)(gridDim.x >> 1);
  const int boxes0 = (p.n_boxes + 1) >> 1;
  const int my_boxes = rank == 0 ? boxes0 : p.n_boxes - boxes0, box0 = rank == 0 ? 0 : boxes0;
  const bool two = p.n_boxes > 1;                                // the second CTA has boxes of its own
  const int cpb = 128 / p.uw;                                    // chunks per box
  const int n_iter = my_boxes == 0 ? 0 : (p.n_tiles - worker + n_workers - 1) / n_workers;
  const uint32_t z_col = (uint32_t)(boxes0 * nb), u_col = p.alias ? z_col : z_col + (uint32_t)nb;

  if (threadIdx.x == 0) {
    for (int i = 0; i < kSlZStages; ++i) { mbar_init(smem_u32(&sh.zf[i]), 1); mbar_init(smem_u32(&sh.ze[i]), 1); }
    mbar_init(smem_u32(&sh.z_full), 1);
    mbar_init(smem_u32(&sh.z_empty), kSlWorkers);
    mbar_init(smem_u32(&sh.g_ready), kSlWorkers);
    for (int i = 0; i < kSlMaxG; ++i) mbar_init(smem_u32(&sh.g_empty[i]), 1);
    for (int i = 0; i < kSlXtStages; ++i) { mbar_init(smem_u32(&sh.xf[i]), 1); mbar_init(smem_u32(&sh.xe[i]), 1); }
    for (int i = 0; i < kSlMaxW; ++i) {
      mbar_init(smem_u32(&sh.wf[i]), 1);
      mbar_init(smem_u32(&sh.wd[i]), kSlWorkers);
      mbar_init(smem_u32(&sh.we[i]), 1);
    }
    for (int i = 0; i < 2; ++i) { mbar_init(smem_u32(&sh.uf[i]), 1); mbar_init(smem_u32(&sh.ue[i]), kSlWorkers); }
    for (int i = 0; i < kSlStaging; ++i) { mbar_init(smem_u32(&sh.sf[i]), kSlWorkers); mbar_init(smem_u32(&sh.se[i]), 1); }
    for (int i = 0; i < kSlPeer; ++i) mbar_init(smem_u32(&sh.peer[i]), 1);
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

  if (warp == 0) {
    // ------------------------------ loads for Z ------------------------------
    uint32_t s = 0, ph = 0;
    bool ok = true;
    for (int i = 0; ok && i < n_iter; ++i) {
      int ci, row0;
      tile_at(i, ci, row0);
      const CUtensorMap* wm = p.w_maps + ci;
      for (int k = 0; k < p.n_boxes; ++k) {
        if (!mbar_wait_warp(smem_u32(&sh.ze[s]), ph ^ 1u, &sh.ctl, p.status, 800 + (int)s)) { ok = false; break; }
        if (elect_one()) {
          const uint32_t bar = smem_u32(&sh.zf[s]), dst = smem_u32(smem_z + s * z_stage);
          mbar_arrive_expect_tx(bar, (uint32_t)z_stage);
          tma_load_2d(dst, wm, bar, k * 128, row0);
          tma_load_2d(dst + kSlBox, &map_x, bar, k * 128, 0);
        }
        __syncwarp();
        if (++s == kSlZStages) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
    const uint32_t idesc_z = make_idesc(128, (uint32_t)nb, 0u, 0u, 0u, 0u);
    const uint32_t idesc_u = make_idesc(128, (uint32_t)p.uw, 1u, 1u, 0u, 0u);
    const uint32_t idesc_g = make_idesc(128, (uint32_t)nb, 1u, 1u, 1u, 1u);
    uint32_t zs = 0, zph = 0, xs = 0, xph = 0, ss = 0, sph = 0, uc = 0;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, int where) {
      if (ok && !mbar_wait_warp(smem_u32(bar), parity, &sh.ctl, p.status, where)) ok = false;
      return ok;
    };
    // boxes [k0, k1) of Z of tile i
    auto issue_z = [&](int i, int k0, int k1) {
      if (k0 == 0 && !wait(&sh.z_empty, (uint32_t)(i & 1) ^ 1u, 810)) return;
      for (int k = k0; k < k1; ++k) {
        if (!wait(&sh.zf[zs], zph, 811)) return;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a = smem_desc_lo(smem_u32(smem_z + zs * z_stage), 16), b = a + (kSlBox >> 4);
#pragma unroll
          for (uint32_t u = 0; u < 4; ++u) umma_f8_lohi(tmem_base + z_col, a + 2u * u, b + 2u * u, desc_hi, idesc_z, (k | (int)u) ? 1u : 0u);
          umma_commit(smem_u32(&sh.ze[zs]));
          if (k + 1 == p.n_boxes) umma_commit(smem_u32(&sh.z_full));
        }
        __syncwarp();
        if (++zs == kSlZStages) { zs = 0; zph ^= 1u; }
      }
    };
    auto issue_gx = [&](int i, int bx, uint32_t g0) {
      if (!wait(&sh.sf[ss], sph, 812)) return;
      tc_fence_after();
      if (elect_one()) {
        // both operands MN-major: blocks of 64 elements kSlBox apart, one MMA eats 16 label rows = 2048 B
        const uint32_t a = smem_desc_lo(smem_u32(smem_s + ss * 2 * kSlBox), kSlBox), b = smem_desc_lo(g0, kSlBox);
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u)
          umma_f16_lohi(tmem_base + (uint32_t)(bx * nb), a + 128u * u, b + 128u * u, desc_hi, idesc_g, (i | (int)u) ? 1u : 0u);
        umma_commit(smem_u32(&sh.se[ss]));
      }
      __syncwarp();
      if (++ss == kSlStaging) { ss = 0; sph ^= 1u; }
    };
    if (n_iter > 0) issue_z(0, 0, p.n_boxes);
    for (int i = 0; ok && i < n_iter; ++i) {
      if (!wait(&sh.g_ready, (uint32_t)(i & 1), 813)) break;
      const int gb = p.g_bufs == 2 ? i & 1 : 0;
      const uint32_t g0 = smem_u32(smem_g + gb * nkb * kSlBox);
      const int n_chunks = my_boxes * cpb;
      int gx_next = 0;
      for (int c = 0; ok && c < n_chunks; ++c, ++uc) {
        const uint32_t ub = uc & 1u, uph = (uc >> 1) & 1u;
        if (!wait(&sh.xf[xs], xph, 814) || !wait(&sh.ue[ub], uph ^ 1u, 815)) break;
        tc_fence_after();
        if (elect_one()) {
          const uint32_t a0 = smem_desc_lo(g0, 16), b0 = smem_desc_lo(smem_u32(smem_xt + xs * xt_stage), 16);
          for (int u = 0; u < nb / 16; ++u) {
            const uint32_t blk = (uint32_t)(u >> 2), in = 2u * (uint32_t)(u & 3);
            umma_f16_lohi(tmem_base + u_col + ub * p.uw, a0 + blk * (kSlBox >> 4) + in, b0 + blk * (uint32_t)(p.uw * 8) + in, desc_hi,
                          idesc_u, u ? 1u : 0u);
          }
          umma_commit(smem_u32(&sh.uf[ub]));
          umma_commit(smem_u32(&sh.xe[xs]));
        }
        __syncwarp();
        if (++xs == kSlXtStages) { xs = 0; xph ^= 1u; }
        // Z of the next tile a few boxes behind every chunk of this one
        if (!p.alias && i + 1 < n_iter) issue_z(i + 1, p.n_boxes * c / n_chunks, p.n_boxes * (c + 1) / n_chunks);
        // gx of a box once the chunk after its last one is under way (its workers are done by then or soon)
        if (c >= cpb + 1 && (c - 1) % cpb == 0) issue_gx(i, gx_next++, g0);
      }
      while (ok && gx_next < my_boxes) issue_gx(i, gx_next++, g0);
      if (ok && elect_one()) umma_commit(smem_u32(&sh.g_empty[gb]));
      __syncwarp();
      if (ok && p.alias && i + 1 < n_iter) {
        // U's last chunks have been read: its columns are Z's again
        for (uint32_t back = 1; back <= 2 && back <= uc; ++back) {
          const uint32_t c = uc - back;
          if (!wait(&sh.ue[c & 1u], (c >> 1) & 1u, 816)) break;
        }
        tc_fence_after();
        if (ok) issue_z(i + 1, 0, p.n_boxes);
      }
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
        if (!mbar_wait_warp(smem_u32(&sh.we[ws]), wph ^ 1u, &sh.ctl, p.status, 820 + (int)ws)) { ok = false; break; }
        if (elect_one()) {
          const uint32_t bar = smem_u32(&sh.wf[ws]);
          mbar_arrive_expect_tx(bar, kSlBox);
          tma_load_2d(smem_u32(smem_w + ws * kSlBox), wm, bar, (box0 + bx) * 128, row0);
        }
        __syncwarp();
        if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
        for (int c = 0; c < cpb; ++c) {
          if (!mbar_wait_warp(smem_u32(&sh.xe[xs]), xph ^ 1u, &sh.ctl, p.status, 830 + (int)xs)) { ok = false; break; }
          if (elect_one()) {
            const uint32_t bar = smem_u32(&sh.xf[xs]), dst = smem_u32(smem_xt + xs * xt_stage);
            mbar_arrive_expect_tx(bar, (uint32_t)xt_stage);
            for (int kb = 0; kb < nkb; ++kb) tma_load_2d(dst + kb * p.uw * 128, &map_xt, bar, kb * 64, (box0 + bx) * 128 + c * p.uw);
          }
          __syncwarp();
          if (++xs == kSlXtStages) { xs = 0; xph ^= 1u; }
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
      if (two && !mbar_wait_warp(smem_u32(&sh.peer[i % kSlPeer]), (uint32_t)(i / kSlPeer) & 1u, &sh.ctl, p.status, 840)) break;
      for (int bx = 0; bx < my_boxes; ++bx) {
        if (!mbar_wait_warp(smem_u32(&sh.wd[ws]), wph, &sh.ctl, p.status, 841)) { ok = false; break; }
        if (lane == 0) {
          tma_store_2d(wm, smem_u32(smem_w + ws * kSlBox), (box0 + bx) * 128, row0);
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
    const int wk = warp - 4, q = warp & 3, h = wk >> 2;
    const int row = q * 32 + lane;                               // label row within the tile
    const uint32_t lane_sel = (uint32_t)(q * 32) << 16;
    const int span = nb >> 2;                                    // batch columns of this warp: [h * span, + span)
    uint32_t* mrow = smem_m + wk * 32;
    uint32_t peer0 = smem_u32(&sh.peer[0]);
    peer0 = mapa_shared(peer0, rank ^ 1u);
    float loss = 0.f;
    uint32_t ws = 0, wph = 0, ss = 0, sph = 0, uc = 0;
    bool ok = true;
    int bkt_beg = 0, bkt_end = 0;
    auto bucket_read = [&](int i) {
      int ci, row0;
      tile_at(i, ci, row0);
      const int bkt = ci * p.bkt_per_chunk + (row0 >> 7);
      bkt_beg = p.bucket_off[bkt];
      bkt_end = p.bucket_off[bkt + 1];
    };
    if (n_iter > 0) bucket_read(0);
    for (int i = 0; ok && i < n_iter; ++i) {
      int ci, row0;
      tile_at(i, ci, row0);
      const int rows = ci == p.n_chunks - 1 ? p.rows_last : p.rows_full;
      const bool row_valid = row0 + row < rows;
      // positives of this warp's rows and columns, one word per row (a duplicate pair counts once)
      uint32_t bits = 0u;
      if (bkt_end > bkt_beg) {
        mrow[lane] = 0u;
        __syncwarp();
        for (int e = bkt_beg + lane; e < bkt_end; e += 32) {
          const uint32_t ent = p.bucket_ent[e];
          const int lrow = (int)(ent >> 16), c = (int)(ent & 0xFFFFu) - h * span;
          if ((lrow >> 5) == q && c >= 0 && c < span) atomicOr(&mrow[lrow & 31], 1u << c);
        }
        __syncwarp();
        bits = mrow[lane];
      }
      if (i + 1 < n_iter) bucket_read(i + 1);
      // --- Z -> G ---
      const int gb = p.g_bufs == 2 ? i & 1 : 0;
      if (!mbar_wait_warp(smem_u32(&sh.z_full), (uint32_t)(i & 1), &sh.ctl, p.status, 850) ||
          !mbar_wait_warp(smem_u32(&sh.g_empty[gb]), (uint32_t)((p.g_bufs == 2 ? i >> 1 : i) & 1) ^ 1u, &sh.ctl, p.status, 851)) {
        ok = false;
        break;
      }
      __syncwarp();
      if (two && wk == 0 && lane == 0) mbar_arrive_remote(peer0 + 8u * (uint32_t)(i % kSlPeer));
      tc_fence_after();
      for (int c8 = 0; c8 < span; c8 += 8) {
        const int b0 = h * span + c8;
        uint32_t v[8], out[4];
        tmem_ld8(tmem_base + lane_sel + z_col + (uint32_t)b0, v);
        tmem_ld_wait_for(v);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int b = b0 + 2 * e;
          const uint32_t zz = pack_bf16x2(__uint_as_float(v[2 * e]) * p.w_scale, __uint_as_float(v[2 * e + 1]) * p.w_scale);
          const float z0 = __uint_as_float(zz << 16), z1 = __uint_as_float(zz & 0xFFFF0000u);
          uint32_t s2 = pack_bf16x2(fast_sigmoid(z0), fast_sigmoid(z1));
          const uint32_t pos = (bits >> (c8 + 2 * e)) & 3u;
          if (pos != 0u) {                                       // bf16(sigmoid) - 1 in bf16 arithmetic
            float lo = __uint_as_float(s2 << 16), hi = __uint_as_float(s2 & 0xFFFF0000u);
            if (pos & 1u) lo = bf16_round(lo - 1.0f);
            if (pos & 2u) hi = bf16_round(hi - 1.0f);
            s2 = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
          }
          if (LOSS && row_valid && rank == 0) {
            if (b < p.batch) loss += bce_softplus(z0) - ((pos & 1u) ? z0 : 0.f);
            if (b + 1 < p.batch) loss += bce_softplus(z1) - ((pos & 2u) ? z1 : 0.f);
          }
          if (!row_valid || b >= p.batch) s2 = 0u;
          else if (b + 1 >= p.batch) s2 &= 0xFFFFu;
          out[e] = s2;
        }
        uint8_t* gp = smem_g + (gb * nkb + (b0 >> 6)) * kSlBox + row * 128 + ((((b0 & 63) >> 3) ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(gp) = make_uint4(out[0], out[1], out[2], out[3]);
      }
      tc_fence_before();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&sh.z_empty));
        mbar_arrive(smem_u32(&sh.g_ready));
      }
      // --- update ---
      const int crow = row0 + row;
      const unsigned long long erow =
          p.upd.elem0 + ((unsigned long long)ci * (unsigned long long)p.rows_full + (unsigned long long)crow) * (unsigned long long)d;
      typename Upd::PhiloxRow pr;
      if (SR) Upd::philox_row(p.upd, (uint32_t)(erow >> 35), pr);
      const bool kahan_row = KAHAN && ci == 0 && crow < p.upd.kahan_rows;
      for (int bx = 0; ok && bx < my_boxes; ++bx) {
        if (!mbar_wait_warp(smem_u32(&sh.wf[ws]), wph, &sh.ctl, p.status, 852) ||
            !mbar_wait_warp(smem_u32(&sh.se[ss]), sph ^ 1u, &sh.ctl, p.status, 853)) {
          ok = false;
          break;
        }
        uint8_t* wbox = smem_w + ws * kSlBox;
        uint8_t* sbox = smem_s + ss * 2 * kSlBox;
        for (int c = 0; c < cpb; ++c, ++uc) {
          const uint32_t ub = uc & 1u, uph = (uc >> 1) & 1u;
          if (!mbar_wait_warp(smem_u32(&sh.uf[ub]), uph, &sh.ctl, p.status, 854)) { ok = false; break; }
          __syncwarp();
          tc_fence_after();
#pragma unroll 1
          for (int half = 0; half < p.uw; half += 64) {
            const int cu = half + 16 * h, cb = c * p.uw + cu;    // column within the chunk, within the box
            const int f0 = (box0 + bx) * 128 + cb;
            uint32_t va[8], vb[8];
            tmem_ld8(tmem_base + lane_sel + u_col + ub * (uint32_t)p.uw + (uint32_t)cu, va);
            tmem_ld8(tmem_base + lane_sel + u_col + ub * (uint32_t)p.uw + (uint32_t)cu + 8u, vb);
            uint4* wslot = ctile_ptr16(wbox, row, cb);
            const uint4 w = *wslot;
            uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
            if (SR) {
              const unsigned long long qq = (erow + (unsigned long long)f0) >> 3;
              if ((uint32_t)(qq >> 32) != pr.q_hi) Upd::philox_row(p.upd, (uint32_t)(qq >> 32), pr);
              ra = Upd::philox(p.upd, pr, (uint32_t)qq);
              rb = Upd::philox(p.upd, pr, (uint32_t)qq + 1u);
            }
            tmem_ld_wait_for(va, vb);
            uint32_t old[8];
            uint4 nw = Upd::update16(p.upd, va, vb, w, ra, rb, old);
            if constexpr (KAHAN) {
              if (kahan_row) {
                uint2 oa = make_uint2(w.x, w.y), ob = make_uint2(w.z, w.w);
                if (row_valid) {
                  const int ks = p.upd.kahan_e5m2 ? 1 : 2;
                  uint8_t* krow = reinterpret_cast<uint8_t*>(p.upd.kahan) + ((size_t)crow * d + f0) * ks;
                  if (f0 < d) oa = Upd::update8_kahan(p.upd, va[0], va[1], va[2], va[3], va[4], va[5], va[6], va[7], oa, ra, krow);
                  if (f0 + 8 < d) ob = Upd::update8_kahan(p.upd, vb[0], vb[1], vb[2], vb[3], vb[4], vb[5], vb[6], vb[7], ob, rb, krow + 8 * ks);
                }
                nw = make_uint4(oa.x, oa.y, ob.x, ob.y);
              }
            }
            *wslot = nw;
            // the old weights as bf16, where the tensor core reads them with the label row as contraction index
            uint8_t* sp = sbox + (cb >> 6) * kSlBox + row * 128;
            const int piece = (cb & 63) >> 3;
            *reinterpret_cast<uint4*>(sp + ((piece ^ (row & 7)) << 4)) = make_uint4(old[0], old[1], old[2], old[3]);
            *reinterpret_cast<uint4*>(sp + (((piece + 1) ^ (row & 7)) << 4)) = make_uint4(old[4], old[5], old[6], old[7]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh.ue[ub]));
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(smem_u32(&sh.wd[ws]));
          mbar_arrive(smem_u32(&sh.sf[ss]));
        }
        if (++ws == (uint32_t)p.w_slots) { ws = 0; wph ^= 1u; }
        if (++ss == kSlStaging) { ss = 0; sph ^= 1u; }
      }
    }
    // --- grad_X: features are lanes, so 32 lanes write 32 neighbouring floats of a batch row ---
    if (ok && n_iter > 0 && mbar_wait_warp(smem_u32(&sh.gx_full), 0u, &sh.ctl, p.status, 855)) {
      __syncwarp();
      tc_fence_after();
      for (int bx = 0; bx < my_boxes; ++bx) {
        const int f = (box0 + bx) * 128 + row;
        for (int c8 = 0; c8 < span; c8 += 8) {
          const int b0 = h * span + c8;
          uint32_t v[8];
          tmem_ld8(tmem_base + lane_sel + (uint32_t)(bx * nb + b0), v);
          tmem_ld_wait_for(v);
          if (f < d) {
            float* dst = p.partial + ((size_t)worker * nb + b0) * d + f;
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (b0 + e < p.batch) dst[(size_t)e * d] = __uint_as_float(v[e]);
          }
          __syncwarp();
        }
      }
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
  cluster_sync_all();                     // the peer may still be arriving on this CTA's barriers
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace xmc
