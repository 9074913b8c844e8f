// grad_X partial sums: partial[split][b][c] (+)= sum over a slice of the chunk's label rows of
// G[l][b] * W[l][c]   (reference: matmul_kernel.py:204-239 large_k_matmul, C = G^T W, operands
// rounded to bf16, fp32 accumulation).
//
// One CTA owns a 256 (batch) x 256 (feature) output tile for one slice of label rows: two 128-lane
// TMEM accumulators of 256 columns.  Both operands are "MN-major" for the tensor core (the
// contraction index, the label row, is the slow index of G[l][b] and W[l][c]), so G tiles land by
// TMA exactly as stored.  e4m3 weights are brought in raw (half the L2 traffic of a bf16 copy and
// no staging pass over HBM) and turned into the bf16 128-byte-swizzled operand layout by the eight
// epilogue warps while the previous stage is being multiplied; after the last stage the same warps
// drain the accumulators.  bf16 weights: after every segment of chain_ksteps stages, so that no accumulator sums
// up more than that (the tensor core truncates; the host's rule has the measurements).  Each (split, tile) owns
// its slot of `partial` and adds to it in the order of the labels: fixed summation order, one writer per element.
//
// PAIR = true: a CTA pair (cluster of two, cta_group::2) owns a tile of HALVES x 256 (batch) x 256 (feature): M = 256
// accumulators of 256 columns, CTA r holding batch rows [256 h + 128 r, +128) of accumulator h in
// its own TMEM.  Each CTA fetches its own HALVES x 128 batch columns of G and only ITS 128 feature columns of
// W (raw, converted by its own warps), so a weight element is converted once per HALVES x 256 batch rows and a
// k-step costs 64 KB of shared-memory traffic per SM for 512 tensor-core cycles instead of 96 KB; the
// smaller stages buy a deeper ring.  Barriers: full lives in the leader (bytes and converter
// warps of both CTAs), mma_done and tmem_full exist in both CTAs and are signalled together by the
// leader's commits, tmem_empty lives in the leader.  Needs d % 256 == 0 (every CTA's half of a feature tile is two whole
// 64-column blocks).  HALVES = 2 is for e4m3 weights and more than 256 batch rows.
//
// bf16 weights on pairs: the accumulator has a twin in TMEM, and a segment is added to sums in the warps' REGISTERS while
// the next one is multiplied; memory sees one store or reduction per launch.  (Emptied into memory by the single-CTA kernel,
// 256 KB of vector reductions a segment, each segment of 512 rows cost 11 000 cycles beside 8 000 of multiplying.)
// grad_X of 131 072 x 768 at batch 256: 73.5 us on single CTAs, 57.3 on pairs.  (Eleven warps are allocated as twelve, which
// leaves a thread 168 registers; with 128 of them sums this kernel spills 28 bytes.)
#pragma once
#include "gemm_engine.cuh"
#include "numerics.cuh"

namespace xmc {

// Label rows per pipeline stage.  The producer's and the issuer's loops take 600 to 700 cycles a stage whatever it
// holds (two waits, three copies, a commit: latencies of a single warp), as much as the tensor core needs for 32
// rows of a 512-row batch tile and twice what it needs for a 256-row one: stages of 32 rows were bound by that.
constexpr int kGxRows = 64;
constexpr int kGxBlockBytes = kGxRows * 128;          // one 64-element block of a stage: 8 KB
constexpr int kGxWarps = 8;
constexpr int kGxThreads = 64 + 32 * kGxWarps + 32;   // producer of G, MMA issuer, converters / drain, producer of raw weights
// per CTA: bf16 feature blocks per stage (a CTA of a pair holds half of the tile's 256 features), ring depths
template <bool PAIR> constexpr int kGxBBlocks = PAIR ? 2 : 4;
template <bool PAIR> constexpr int kGxBBytes = kGxBBlocks<PAIR> * kGxBlockBytes;       // 16 / 32 KB
// Blocks of 64 batch columns per CTA and stage, raw e4m3 bytes, ring depths.  bf16 weights arrive as the operand; the single
// CTA keeps the raw ring's place for the drain's staging tiles.
template <bool CONVERT, bool PAIR, int HALVES>
struct GxShape {
  static constexpr int kABlocks = PAIR ? 2 * HALVES : 4, kABytes = kABlocks * kGxBlockBytes;
  static constexpr int kRawBytes = PAIR && !CONVERT ? 0 : kGxBBlocks<PAIR> * kGxRows * 64;   // 8 / 16 KB
  static constexpr int kStages = !PAIR ? 3 : !CONVERT ? 6 : HALVES == 2 ? 4 : 5;
  static constexpr int kRawStages = !PAIR ? 2 : !CONVERT ? 0 : kStages;
  static constexpr int kSmemBytes = kStages * (kABytes + kGxBBytes<PAIR>) + kRawStages * kRawBytes;
};
constexpr int kGxMaxStages = 6;

struct GxParams {
  int bpad, d;
  int n_btiles, n_dtiles, n_splits;   // batch tiles of 256, feature tiles of 256
  int total_ksteps;                   // stages of kGxRows label rows of G in this launch
  const CUtensorMap* w_maps;          // one per weight chunk, in device memory; nullptr: the kernel's own map_w for all rows
  int first_kstep;                    // weight side: stage 0 of this launch in the list of all chunks' stages ...
  int ksteps_per_chunk;               // ... of which every chunk but the last has this many
  int accumulate;                     // 0: overwrite the slot (first chunk of a step)
  int chain_ksteps;                   // bf16 weights: stages that an accumulator sums up before it is added to the slot
  float* partial;                     // [n_splits][bpad][d]
  int* status;
};

struct GxShared {
  uint64_t full[kGxMaxStages];          // the stage's G tile has landed and its weight block has been converted (or landed)
  uint64_t mma_done[kGxMaxStages];      // the MMAs reading stage s have completed
  uint64_t raw_full[kGxMaxStages];
  uint64_t raw_empty[kGxMaxStages];
  uint64_t tmem_full[2], tmem_empty[2]; // a segment has been multiplied / drained, per accumulator set
  uint32_t tmem_base;
  Ctl ctl;
};

template <bool CONVERT, bool PAIR, int HALVES>
constexpr int kGxSmemBytes = GxShape<CONVERT, PAIR, HALVES>::kSmemBytes + (int)sizeof(GxShared) + 1024;

template <bool CONVERT, bool PAIR = false, int HALVES = 2>
__global__ void __launch_bounds__(kGxThreads, 1)
gradx_kernel(const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_w,
             const GxParams p) {
  using Shape = GxShape<CONVERT, PAIR, HALVES>;
  constexpr int kStages = Shape::kStages, kRawStages = Shape::kRawStages, kABytes = Shape::kABytes;
  constexpr int kBBytes = kGxBBytes<PAIR>, kRawBytes = Shape::kRawBytes, kBBlocks = kGxBBlocks<PAIR>;
  static_assert(HALVES == 2 || (PAIR && HALVES == 1), "a single CTA has 256 batch rows as two accumulators of 128 lanes");
  static_assert(kStages <= kGxMaxStages && kGxSmemBytes<CONVERT, PAIR, HALVES> <= 232448, "exceeds the shared memory a CTA can get");
  constexpr bool kRegSums = PAIR && !CONVERT;          // segments add up in registers, accumulator sets alternate
  static_assert(!kRegSums || HALVES == 1, "two accumulators fill TMEM");
  static_assert(PAIR || CONVERT || kRawStages * kRawBytes >= kGxWarps * 4096, "the drain's staging tiles lie in the raw ring");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* smem_a = smem;                                         // [stage][4 blocks][64 rows][128 B]
  uint8_t* smem_b = smem + kStages * kABytes;                     // [stage][2 or 4 blocks][64 rows][128 B], bf16 weights
  uint8_t* smem_r = smem_b + kStages * kBBytes;                   // [raw stage][blocks][64 rows][64 B] e4m3
  GxShared& sh = *reinterpret_cast<GxShared*>(smem_r + kRawStages * kRawBytes);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  static_assert(kGxWarps == 8 && kGxRows % 32 == 0, "converter mapping assumes 8 warps and bands of 8 rows");
  uint32_t rank = 0u;
  if constexpr (PAIR) rank = cluster_ctarank();

  // tile coordinates: n_btiles counts batch tiles of 256 (single CTA) or HALVES x 256 (pair)
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int per = p.n_btiles * p.n_dtiles;
  const int split = worker / per;
  const int rem = worker - split * per;
  const int bt = rem / p.n_dtiles, dt = rem - bt * p.n_dtiles;
  const int b0 = bt * (PAIR ? HALVES * 256 : 256), c0 = dt * 256;
  // A split's slice is every n_splits-th stage, last one first: the kernel as a whole walks G and the weights once, from
  // where the forward kernel ended -- what that left in L2 is read before it is pushed out -- to where the update
  // begins.  (Slices of consecutive rows, each from its first one on: e4m3 75 776 x 768 launches at batch 512, grad_X 45.1 us
  // where this takes 43.0; bf16 131 072 x 768 at 256 57.3 and 55.4; the updates behind them 1 % more.)
  const int k_steps = split < p.total_ksteps ? (p.total_ksteps - 1 - split) / p.n_splits + 1 : 0;
  const int k_first = p.total_ksteps - 1 - split;
  const int n_eff = PAIR ? 256 : min(256, (p.d - c0 + 15) & ~15);
  // Segments of the slice, each summed in the accumulators from zero.  (e4m3 weights: always one, see chain_ksteps.)
  const int n_segs = CONVERT ? 1 : max(1, (k_steps + p.chain_ksteps - 1) / p.chain_ksteps);
  auto seg_end = [&](int seg) { return (int)((long long)k_steps * (seg + 1) / n_segs); };
  // where the slice's stages lie among the weight chunks
  int w_chunk = max(0, p.first_kstep + k_first) / p.ksteps_per_chunk;
  int w_step = p.first_kstep + k_first - w_chunk * p.ksteps_per_chunk;
  auto w_map = [&]() { return p.w_maps != nullptr ? p.w_maps + w_chunk : &map_w; };
  auto w_next = [&]() {
    for (w_step -= p.n_splits; w_step < 0 && w_chunk > 0; --w_chunk) w_step += p.ksteps_per_chunk;
  };
  // accumulators in use, and this CTA's 128 batch rows of accumulator h: [b_cta + h * b_half, +128)
  const int m_halves = PAIR ? ((HALVES == 2 && b0 + 256 < p.bpad) ? 2 : 1) : ((b0 + 128 < p.bpad) ? 2 : 1);
  const int b_half = PAIR ? 256 : 128;
  const int b_cta = b0 + (PAIR ? 128 * (int)rank : 0);
  const int c_cta = c0 + (PAIR ? 128 * (int)rank : 0);           // first feature column this CTA stages

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      // bytes of G, weights (converted, or bytes announced by their producer)
      mbar_init(smem_u32(&sh.full[s]), 1 + (CONVERT ? (PAIR ? 2 : 1) * kGxWarps : PAIR ? 1 : 0));
      mbar_init(smem_u32(&sh.mma_done[s]), 1);
    }
    for (int s = 0; s < kRawStages; ++s) {
      mbar_init(smem_u32(&sh.raw_full[s]), 1);
      mbar_init(smem_u32(&sh.raw_empty[s]), kGxWarps);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&sh.tmem_full[b]), 1);
      mbar_init(smem_u32(&sh.tmem_empty[b]), (PAIR ? 2 : 1) * kGxWarps);
    }
    sh.ctl.abort = 0;
    sh.ctl.limit = kWaitLimitCycles;
    fence_barrier_init();
    tma_prefetch_desc(&map_g);
    tma_prefetch_desc(&map_w);
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(smem_u32(&sh.tmem_base), kTmemCols);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(&sh.tmem_base), kTmemCols);
      tmem_relinquish();
    }
  }
  constexpr int kWProducer = CONVERT || PAIR ? 2 + kGxWarps : 0;        // the warp that fetches weights
  if (warp == kWProducer && p.w_maps != nullptr)
    tensormap_acquire(p.w_maps, p.first_kstep / p.ksteps_per_chunk, (p.first_kstep + p.total_ksteps - 1) / p.ksteps_per_chunk);
  pdl_launch_dependents();                  // the next kernel may start its prologue as SMs free up
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // both CTAs' barriers exist before anything remote happens
  else __syncthreads();
  // The weights depend on nothing before this kernel (they were last written a step ago): a producer of their own starts at
  // once, everybody else waits for the kernel that writes G.
  if (kWProducer == 0 || warp != kWProducer) pdl_wait();
  tc_fence_after();
  const uint32_t tmem_base = sh.tmem_base;
  // barriers the two CTAs of a pair share live in the leader
  uint32_t full0 = smem_u32(&sh.full[0]);
  if constexpr (PAIR) full0 = mapa_shared(full0, 0);

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    // The whole warp runs the loop on warp-uniform values (uniform registers: the TMA instructions take
    // their operands there) and one elected lane issues; ring indices are running counters.
    {
      uint32_t s = 0, ph = 0;
      int krow = k_first * kGxRows;
      for (int i = 0; i < k_steps; ++i, krow -= p.n_splits * kGxRows) {
        if (!mbar_wait_warp(smem_u32(&sh.mma_done[s]), ph ^ 1u, &sh.ctl, p.status, 510 + (int)s)) break;
        if (elect_one()) {
          const uint32_t sa = smem_u32(smem_a + s * kABytes);
          if constexpr (PAIR) {
            // this CTA's 128 batch columns of either accumulator in use: boxes [2 blocks][64 rows][128 B];
            // the bytes of both CTAs are counted on the leader's barrier
            if (rank == 0) mbar_arrive_expect_tx(smem_u32(&sh.full[s]), m_halves * 4 * kGxBlockBytes);
            const uint32_t ab = full0 + 8u * s;
            tma_load_3d_pair(sa, &map_g, ab, 0, krow, b_cta >> 6);
            if (HALVES == 2 && m_halves == 2) tma_load_3d_pair(sa + 2 * kGxBlockBytes, &map_g, ab, 0, krow, (b_cta + 256) >> 6);
          } else {
            const uint32_t ab = smem_u32(&sh.full[s]);
            mbar_arrive_expect_tx(ab, kABytes + (CONVERT ? 0 : kBBytes));
            // one box: [4 batch blocks][64 rows][128 B], blocks beyond the batch are zero-filled
            tma_load_3d(sa, &map_g, ab, 0, krow, b0 >> 6);
            if constexpr (!CONVERT) tma_load_3d(smem_u32(smem_b + s * kBBytes), w_map(), ab, 0, w_step * kGxRows, c0 >> 6);
          }
        }
        __syncwarp();
        if constexpr (kWProducer == 0) w_next();
        if (++s == (uint32_t)kStages) { s = 0; ph ^= 1u; }
      }
    }
  } else if (kWProducer != 0 && warp == kWProducer) {
    // ------------------------------ TMA producer of weights: raw tiles, or the operand itself ------------------------------
    // A warp of its own: the two waits and copies of a stage took one warp about 750 cycles, and the tensor core waited for
    // it (e4m3, 131 072 x 768 at batch 256: 60.3 -> 52.8 us).
    uint32_t s = 0, ph = 0;
    constexpr uint32_t kRing = CONVERT ? kRawStages : kStages;
    for (int i = 0; i < k_steps; ++i) {
      if (!mbar_wait_warp(smem_u32(CONVERT ? &sh.raw_empty[s] : &sh.mma_done[s]), ph ^ 1u, &sh.ctl, p.status, 500 + (int)s)) break;
      if (elect_one()) {
        // one box: [feature blocks][64 rows][64 or 128 B]
        if constexpr (CONVERT) {
          const uint32_t rb = smem_u32(&sh.raw_full[s]);
          mbar_arrive_expect_tx(rb, kRawBytes);
          tma_load_3d(smem_u32(smem_r + s * kRawBytes), w_map(), rb, 0, w_step * kGxRows, c_cta >> 6);
        } else {
          if (rank == 0) mbar_arrive_expect_tx(smem_u32(&sh.full[s]), 2 * kBBytes);
          tma_load_3d_pair(smem_u32(smem_b + s * kBBytes), w_map(), full0 + 8u * s, 0, w_step * kGxRows, c_cta >> 6);
        }
      }
      __syncwarp();
      w_next();
      if (++s == kRing) { s = 0; ph ^= 1u; }
    }
    // whoever runs behind this kernel relies on every role having waited for the one before
    pdl_wait();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (of a pair: the leader's) ------------------------------
    if (!PAIR || rank == 0) {
      const uint32_t idesc = make_idesc(PAIR ? 256 : 128, (uint32_t)n_eff, 1u, 1u, 1u, 1u);
      // MN-major, 128B swizzle: 64-element blocks kGxBlockBytes apart (leading offset), 8-row
      // groups 1024 B apart (stride offset); one UMMA consumes 16 label rows = 2048 B per block
      constexpr uint32_t desc_hi = smem_desc_hi_sw128(1024);
      const uint32_t a_lo0 = smem_desc_lo(smem_u32(smem_a), kGxBlockBytes);
      const uint32_t b_lo0 = smem_desc_lo(smem_u32(smem_b), kGxBlockBytes);
      bool ok = true;
      uint32_t s = 0, ph = 0;
      for (int seg = 0, i = 0; ok && seg < n_segs; ++seg) {
        // the set's last segment has been read: the one before, or with alternating sets the one before that
        const int set = kRegSums ? seg & 1 : 0, turn = kRegSums ? seg >> 1 : seg;
        const uint32_t d_tmem = tmem_base + (uint32_t)set * 256u;
        if (turn > 0) {
          if (!mbar_wait_warp(smem_u32(&sh.tmem_empty[set]), (uint32_t)(turn - 1) & 1u, &sh.ctl, p.status, 530)) break;
          tc_fence_after();
        }
        uint32_t acc = 0u;
        for (const int end = seg_end(seg); i < end; ++i) {
          if (!mbar_wait_warp(smem_u32(&sh.full[s]), ph, &sh.ctl, p.status, 520 + (int)s)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            const uint32_t a_lo = a_lo0 + s * (uint32_t)(kABytes >> 4), b_lo = b_lo0 + s * (uint32_t)(kBBytes >> 4);
            for (int hm = 0; hm < m_halves; ++hm) {
#pragma unroll
              for (uint32_t u = 0; u < kGxRows / 16; ++u) {
                // accumulator hm reads this CTA's (of a pair: either CTA's) blocks 2 hm, 2 hm + 1 of the G stage
                const uint32_t au = a_lo + (uint32_t)hm * (2u * kGxBlockBytes >> 4) + 128u * u, bu = b_lo + 128u * u;
                if constexpr (PAIR) umma_f16_lohi_pair(d_tmem + hm * 256, au, bu, desc_hi, idesc, u == 0 ? acc : 1u);
                else umma_f16_lohi(d_tmem + hm * 256, au, bu, desc_hi, idesc, u == 0 ? acc : 1u);
              }
            }
            if constexpr (PAIR) umma_commit_pair(smem_u32(&sh.mma_done[s]));
            else umma_commit(smem_u32(&sh.mma_done[s]));
          }
          __syncwarp();
          acc = 1u;
          if (++s == (uint32_t)kStages) { s = 0; ph ^= 1u; }
        }
        if (ok && elect_one()) {
          if constexpr (PAIR) umma_commit_pair(smem_u32(&sh.tmem_full[set]));
          else umma_commit(smem_u32(&sh.tmem_full[set]));
        }
        __syncwarp();
      }
    }
  } else if (warp < 2 + kGxWarps) {
    // -------------------- converters, then epilogue (warps 2..9) --------------------
    const int cw = warp - 2;                                      // 0..7
    const int q = warp & 3;
    const int hm = cw >> 2;                                       // warps 2..5 -> accumulator (of one: columns) 0, 6..9 -> 1
    const bool have_acc = k_steps > 0;
    // 32 columns of this warp's 32 rows into the slot, from column cg of its share on.  Through a per-warp 32 x 32 staging
    // tile so that the global accesses run along rows: 8 lanes cover 128 contiguous bytes of one batch row instead of 32
    // lanes touching 32 different rows with 16 bytes each.  The tiles lie in the raw ring where nothing arrives raw, else in
    // the operand stages, idle by then.
    const int brow0 = b_cta + (HALVES == 2 ? hm * b_half : 0) + q * 32;       // first batch row of this warp
    const int ccol0 = c0 + (HALVES == 2 ? 0 : hm * 128);                      // first feature
    float* dst0 = p.partial + ((size_t)split * p.bpad + brow0) * p.d + ccol0;
    float4* stage = reinterpret_cast<float4*>((CONVERT || PAIR ? smem_a : smem_r) + cw * 4096);   // [32 rows][8 chunks of 16 B], XOR-swizzled
    const int rr = lane >> 3, ch = lane & 7;                                  // read side: row within a group of 4, 16-byte chunk
    auto drain = [&](int cg, const uint32_t (&v)[32], bool accumulate) {
      __syncwarp();                                               // the previous group's reads are done
#pragma unroll
      for (int i = 0; i < 8; ++i)
        stage[lane * 8 + (i ^ (lane & 7))] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                                         __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
      __syncwarp();
      const bool col_ok = ccol0 + cg + 4 * ch < p.d;              // d is a multiple of 4
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = 4 * j + rr;
        const float4 o = stage[r * 8 + (ch ^ (r & 7))];
        if (!col_ok || brow0 + r >= p.bpad || (HALVES == 2 && hm >= m_halves)) continue;
        float4* ptr = reinterpret_cast<float4*>(dst0 + (size_t)r * p.d + cg + 4 * ch);
        if (accumulate) {
          // Fire-and-forget vector reduction at L2: no read latency here.  Each element has exactly one
          // thread that writes it, in order, and launches are stream-ordered: the order of additions is fixed.
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(ptr), "f"(o.x), "f"(o.y),
                       "f"(o.z), "f"(o.w)
                       : "memory");
        } else {
          *ptr = o;
        }
      }
    };
    uint32_t empty0 = smem_u32(&sh.tmem_empty[0]);
    if constexpr (PAIR) empty0 = mapa_shared(empty0, 0);
    float sums[kRegSums ? 128 : 1];
    if constexpr (kRegSums) {
#pragma unroll
      for (int i = 0; i < 128; ++i) sums[i] = 0.f;
    }
    bool ok = true;
    uint32_t s = 0, ph = 0, rs = 0, rph = 0;
    for (int seg = 0, i = 0; ok && seg < n_segs; ++seg) {
      if constexpr (CONVERT) {
        for (const int end = seg_end(seg); i < end; ++i) {
          if (!mbar_wait(smem_u32(&sh.raw_full[rs]), rph, &sh.ctl, p.status, 540 + (int)rs) ||
              !mbar_wait(smem_u32(&sh.mma_done[s]), ph ^ 1u, &sh.ctl, p.status, 550 + (int)s)) {
            ok = false;
            break;
          }
          // A warp takes one 64-feature block and a band of rows; per pass 8 rows x 64 B of the block: the
          // reads are one contiguous 512 B run, the swizzled writes hit every bank equally often.
          // Single CTA: 4 blocks x 2 bands of 32 rows (4 passes); pair: 2 blocks x 4 bands of 16 rows (2 passes).
          constexpr int kBands = kGxWarps / kBBlocks, kPasses = kGxRows / (8 * kBands);
          const int blk = cw % kBBlocks, band = cw / kBBlocks;
          const uint8_t* raw = smem_r + rs * kRawBytes + blk * (kGxRows * 64);
          uint8_t* dst = smem_b + s * kBBytes + blk * kGxBlockBytes;
#pragma unroll
          for (int it = 0; it < kPasses; ++it) {
            const int row = 8 * (kPasses * band + it) + (lane >> 2), kc = lane & 3;
            const uint4 v = *reinterpret_cast<const uint4*>(raw + row * 64 + kc * 16);
            uint4 o0, o1;
            e4m3x4_to_bf16x4(v.x, o0.x, o0.y);
            e4m3x4_to_bf16x4(v.y, o0.z, o0.w);
            e4m3x4_to_bf16x4(v.z, o1.x, o1.y);
            e4m3x4_to_bf16x4(v.w, o1.z, o1.w);
            uint8_t* rowp = dst + row * 128;
            *reinterpret_cast<uint4*>(rowp + (((2 * kc) ^ (row & 7)) << 4)) = o0;
            *reinterpret_cast<uint4*>(rowp + (((2 * kc + 1) ^ (row & 7)) << 4)) = o1;
          }
          fence_proxy_async();                                      // generic-proxy writes -> tensor-core reads
          __syncwarp();                                             // one arrival per warp: 256 arrivals on one
          if (lane == 0) {                                          // barrier word would serialise the stage
            if constexpr (PAIR) mbar_arrive_remote(full0 + 8u * s);    // the leader's barrier counts the warps of both CTAs
            else mbar_arrive(full0 + 8u * s);
            mbar_arrive(smem_u32(&sh.raw_empty[rs]));
          }
          if (++s == (uint32_t)kStages) { s = 0; ph ^= 1u; }
          if (++rs == (uint32_t)kRawStages) { rs = 0; rph ^= 1u; }
        }
      }
      const int set = kRegSums ? seg & 1 : 0, turn = kRegSums ? seg >> 1 : seg;
      if (!ok || !mbar_wait(smem_u32(&sh.tmem_full[set]), (uint32_t)turn & 1u, &sh.ctl, p.status, 560)) { ok = false; break; }
      __syncwarp();
      tc_fence_after();
      if constexpr (kRegSums) {
        // the set's columns are free as soon as they are in registers
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(set * 256 + hm * 128);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t v[32];
          if (have_acc) {
            tmem_ld32(taddr + 32 * g, v);
            tmem_ld_wait_for(v);
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) v[e] = 0u;
          }
#pragma unroll
          for (int e = 0; e < 32; ++e) sums[32 * g + e] += __uint_as_float(v[e]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(empty0 + 8u * (uint32_t)set);
      } else {
        const bool accumulate = p.accumulate || seg > 0;
        if (have_acc || !accumulate) {
          const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(HALVES == 2 ? hm * 256 : hm * 128);
          for (int cg = 0; cg < (HALVES == 2 ? n_eff : 128); cg += 32) {
            uint32_t v[32];
            if (have_acc && (HALVES == 1 || hm < m_halves)) {
              tmem_ld32(taddr + cg, v);
              tmem_ld_wait();
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = 0u;
            }
            drain(cg, v, accumulate);
          }
        }
        if (seg + 1 < n_segs) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&sh.tmem_empty[0]));
        }
      }
    }
    if constexpr (kRegSums) {
      if (ok && (have_acc || !p.accumulate)) {
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t v[32];
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(sums[32 * g + e]);
          drain(32 * g, v, p.accumulate != 0);
        }
      }
    }
  }

  __syncwarp();
  if (sh.ctl.abort) {
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();   // the peer may still be reading this CTA's shared memory or arriving on its barriers
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, kTmemCols);
    else tmem_dealloc(tmem_base, kTmemCols);
  }
}

}  // namespace xmc
