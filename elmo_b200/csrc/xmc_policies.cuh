// GEMM policies (tile mapping + epilogue) of the chunked XMC step:
//   FwdPolicy    Z^T[labels x batch] = W X^T  ->  G = sigmoid(Z) - Y  (bf16, label-major), loss terms
//   UpdPolicy    acc[labels x d] = G X        ->  W <- round(W - lr*(acc + wd*W))   (dW never stored)
//   LogitsPolicy out[batch x labels] = bf16(X W^T)  (inference forward)
//   PlainPolicy  D = A B^T (engine self-test)
#pragma once
#include "gemm_engine.cuh"
#include "numerics.cuh"

namespace xmc {

__device__ __forceinline__ int round_up16(int v) { return (v + 15) & ~15; }

// x / d by one multiply: the roles recompute their tile coordinates once per tile, and a real division (its
// reciprocal comes from the special-function pipe the forward epilogue saturates) put hundreds of cycles between
// two tiles.  mul = floor(2^32 / d) + 1, exact for x * d < 2^32; 0 for d == 1; 1 (a real division) where the
// largest x is too large for it.
struct FastDiv {
  uint32_t mul;
  int d;
};
__host__ __device__ inline FastDiv make_fastdiv(int d, long long largest) {
  FastDiv f;
  f.d = d;
  f.mul = d <= 1 ? 0u : largest * d >= 0x100000000ll ? 1u : (uint32_t)(0x100000000ull / (unsigned long long)d) + 1u;
  return f;
}
__device__ __forceinline__ int fast_div(int x, const FastDiv& f) {
  return f.mul == 0u ? x : f.mul == 1u ? x / f.d : (int)__umulhi((uint32_t)x, f.mul);
}

// The label rows of a handle as one list of tiles, every weight chunk padded to whole tiles; a launch takes a run of
// them, across chunks.  (One launch per chunk paid each kernel's ramp and half-empty last round once per chunk.)
struct LabelTiles {
  int m_rows;                // rows of a tile
  FastDiv per_chunk;         // tiles of a chunk (of every one but the last, which may have fewer)
  int rows_full, rows_last;  // label rows of every chunk but the last, of the last
  int n_chunks;
  int first, count;          // this launch: tiles [first, first + count)
  __device__ __forceinline__ int chunk_of(int rel) const { return fast_div(first + rel, per_chunk); }
  __device__ __forceinline__ void locate(int rel, Job& j, int& row0) const {
    const int t = first + rel;
    j.chunk = chunk_of(rel);
    row0 = (t - j.chunk * per_chunk.d) * m_rows;
    j.rows = j.chunk == n_chunks - 1 ? rows_last : rows_full;
  }
  __device__ __forceinline__ long long row_of(const Job& j, int row) const { return (long long)j.chunk * rows_full + row; }
};

struct NoState {};

// f(entry) for the positives ents[beg, end) of a bucket, by the lanes of a warp, AHEAD loads of a lane in flight.  Popular
// labels share a bucket -- sorted by popularity, the first 128 of 2.8 million labels have half of a step's 30 000 pairs --
// and a loop that waits for each load walks it at 32 pairs a trip to L2 while the other tiles' warps are long done.
// First forward launch of 2 812 281 x 768, batch 1024, 245 -> 110 us (those behind it 72); of 500 000 x 768 simulated FP8,
// batch 256, 81 -> 59 (58).
template <int AHEAD, class F>
__device__ __forceinline__ void for_each_entry(const uint32_t* __restrict__ ents, int beg, int end, int lane, F&& f) {
  for (int e0 = beg + lane; e0 < end; e0 += 32 * AHEAD) {
    uint32_t ent[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) ent[u] = e0 + 32 * u < end ? ents[e0 + 32 * u] : 0xFFFFFFFFu;   // no entry has bit 31
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (!(ent[u] >> 31)) f(ent[u]);
  }
}

// -------------------------------------------------------------------------------------------------
// Forward + loss-gradient epilogue.
// Reference arithmetic reproduced here: logits rounded to bf16 (output dtype of torch._scaled_mm /
// torch.matmul, chunked_fp8xmc_clf.py:98-102), sigmoid rounded to bf16 (:107), "-1" applied in bf16 at
// the positives with set semantics (:108).
// -------------------------------------------------------------------------------------------------
struct FwdParams {
  int after_prep;          // X was written by the kernel before this one, or by the caller's: every role waits for it
  LabelTiles lt;
  const CUtensorMap* w_maps;   // one per chunk, in device memory
  int n_btiles;            // batch tiles of 256
  FastDiv div_btiles;      // of n_btiles
  int batch, bpad;         // valid batch rows, padded row length of G (multiple of 16)
  int x_rows;              // rows of a box of X
  int k_steps;             // cdiv(d * elem_size, 128)
  float w_scale;
  const float* x_scale;    // split embeddings: w_scale over the power of two that a batch row was multiplied by
  int part_rows;           // ... rows from one part of X to the next
  const uint8_t* x_wide;   // ... which batch rows are wide (PrepX), or nullptr
  __nv_bfloat16* G;        // [lt.count * lt.m_rows x bpad]
  uint8_t* G8;             // WRITE_G8 variants: e4m3(G * 256), same shape (operand of the FP8 dW contraction)
  const int* bucket_off;   // positives bucketed by label tile: offsets ...
  const uint32_t* bucket_ent;  // ... entries: batch row | (label-in-tile << 16)
  int bkt_per_chunk;       // buckets (128 label rows each) of a chunk
  double* loss_partial;    // [gridDim.x * kEpiWarps] or nullptr
  int* status;
};

constexpr float kG8Scale = 256.0f;      // |G| < 1: e4m3(G * 256) stays below 448

// How the logits of e4m3 weights and bf16 embeddings are multiplied, "simulated FP8": the embeddings in two parts on the FP8 tensor
// cores (PrepX), or the weights converted to bf16 in shared memory by the engine's converter warps, which takes them 1000 cycles for
// 64 features where the tensor core needs 500 either way.  Split, a product has at most eight significant bits and is exact, as the
// bf16 one, for what the parts hold exactly: all that is above 2^-13 of a row's largest, in a wide row 2^-23; what they lack of a row
// is no more than 2^-24 of its magnitudes, summed up.  The sums are fp32 as there: relative 2-norm error of the logits against 64 bits, weights U(+-1/sqrt(d)), 3.5e-8 and
// 3.5e-8 with 768 features, 1.6e-8 and 1.7e-8 with 384, 4.0e-8 and 4.1e-8 with 1 024; weights over ten binades 7.1e-7 and 6.2e-7.
// Steps with the forward converted and split, three kernels, us in a loop: 500 000 x 768 at batch 40 520 and 467, 256 764 and 724, with the loss at
// 64 550 and 482; 400 000 x 256 with the loss at 200 366 and 324; 1 000 000 x 64 at 64 270 and 257, 256 480 and 487, with the loss 733 and 623.
enum Simulated { kSimNone, kSimConvert, kSimSplit };

// what the accumulators of four batch rows are multiplied by, two and two.  (Volatile: asked for all at once the 32 of a column group cost
// more registers than there are.)
__device__ __forceinline__ void shared_scales(uint32_t at, uint64_t (&two)[2]) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(two[0]), "=l"(two[1]) : "r"(at));
}
// bf16 logits of two batch rows
__device__ __forceinline__ uint32_t scaled_bf16x2(uint32_t v0, uint32_t v1, uint64_t scales) {
  float z0, z1;
  unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(v0), __uint_as_float(v1)), scales), z0, z1);
  return pack_bf16x2(z0, z1);
}

// SPLIT: bf16 embeddings in two parts, of tiles with a wide row four (PrepX), by e4m3 weights.
template <bool FP8, bool LOSS, bool WRITE_G8 = false, bool SPLIT = false>
struct FwdPolicy {
  static_assert(FP8 || !SPLIT, "the parts are FP8 operands");
  using Params = FwdParams;
  static constexpr bool kMnMajor = false;
  static constexpr bool kChunkMaps = true;   // Params::w_maps are the maps of one operand or of the epilogue's tile
  static constexpr bool kFp8 = FP8;
  static constexpr uint32_t kFmt = FP8 ? 0u : 1u;            // e4m3 | bf16
  static constexpr int kElemsPerRow = FP8 ? 128 : 64;
  static constexpr int kEpiWarps = 16;
  // FP8: G leaves through shared memory by TMA, a box of 32 label rows x 64 batch columns per warp, paid for with
  // two operand stages (forward of 300 000 x 768, batch 2048: 755 -> 690 us; batch 256: no change).  bf16 operands take twice
  // the stages per feature and miss them more (+4 to +10 %): there the threads store 64 bytes of their row.
  static constexpr bool kTmaG = FP8 && !SPLIT;
  static constexpr int kStages = SPLIT ? 2 : kTmaG ? 3 : 4;
  static constexpr int kStagesPair = kTmaG || SPLIT ? 4 : 6;
  static constexpr int kSplit = SPLIT ? 2 : 0, kXRows = 2;
  __device__ static int x_rows(const Params& p) { return p.x_rows; }
  __device__ static int tile_rows(const Params&) { return kTileN; }       // batch rows of a tile
  __device__ static int x_tile(const Job& j) { return j.t1; }
  static constexpr bool kConv = false, kEarlyWeights = false;
  static constexpr bool kCTile = false;
  static constexpr int kCBufs = 1;
  static constexpr int kCParts = 1;
  static constexpr bool kBitmap = true;
  static constexpr int kEpiStage = kTmaG ? 4096 : SPLIT ? 256 : 0;      // a box of G; the scales of the warp's columns, 64 at most
  // W of this chunk was last written a step ago and the quantised X, but for the first launch of a step, by a
  // kernel that others which waited for it separate from this one: the operand loads need not wait for the kernels
  // before.  The epilogue overwrites G, which the previous chunk's kernels read: it waits.
  static constexpr int kWaitRoles = kRoleEpilogue | kRoleExtra;
  __device__ static bool wait_all(const Params& p) { return p.after_prep != 0; }
  __device__ static long long wait_limit(const Params&) { return kWaitLimitCycles; }
  __device__ static bool skip_load(const Params&, int, int) { return false; }
  struct EpilogueState {
    float loss;
    int has_pos;
    int next_bkt, next_beg, next_end;   // bucket range of the CTA's next tile, read a tile ahead
    int scales_of;                      // the batch tile whose scales the warp has in shared memory
  };

  __device__ static const CUtensorMap* map_a(const Params& p, const Job& j, const CUtensorMap*) { return p.w_maps + j.chunk; }
  __device__ static const CUtensorMap* map_b(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_c(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static int num_tiles(const Params& p) { return p.lt.count * p.n_btiles; }
  __device__ static void job(const Params& p, int tile, Job& j) {
    j.t0 = fast_div(tile, p.div_btiles);   // label tile
    j.t1 = tile - j.t0 * p.n_btiles;   // batch tile
    p.lt.locate(j.t0, j, j.a0);
    j.c_row = j.t0 * p.lt.m_rows;      // row of G
    j.b0 = j.t1 * kTileN;
    j.k_begin = 0;
    j.k_steps = p.k_steps;
    j.n_eff = min(kTileN, round_up16(p.bpad - j.b0));
  }
  __device__ static void epilogue_begin(const Params&, EpilogueState& st) {
    st.loss = 0.f;
    st.has_pos = 0;
    st.next_bkt = -1;
    st.next_beg = st.next_end = 0;
    st.scales_of = -1;
  }
  // The bucket offsets are two dependent-free global reads whose latency would otherwise sit between two
  // epilogues (the epilogue warps are the busiest role of this kernel): issue them one tile ahead.
  __device__ static void epilogue_prefetch(const Params& p, const Job& jn, EpilogueState& st) {
    st.next_bkt = -1;
    if (jn.a0 >= jn.rows) return;
    st.next_bkt = jn.chunk * p.bkt_per_chunk + (jn.a0 >> 7);
    st.next_beg = p.bucket_off[st.next_bkt];
    st.next_end = p.bucket_off[st.next_bkt + 1];
  }
  // log2 of the neighbouring columns a warp takes: with the loss, and of split embeddings, an equal share of the tile's, down to 32 -- its
  // epilogue is what the kernel waits for -- and with both down to 16: up to batch 64 half of the warps did it (step of 1 000 000 x 64 at 64, three kernels,
  // 343 and 305 us).  Else,
  // and with G stored by TMA in lines of 64, of all 256: shares change nothing there up to batch 64 and cost 4 % of the forward at 100.
  __device__ static int col_shift(const Job& j) {
    static_assert(kTileN == (kEpiWarps / 4) << 6, "four warps share a row");
    if constexpr (kTmaG || !(LOSS || SPLIT)) return 6;
    int sh = 6;
    while (sh > (SPLIT && LOSS ? 4 : 5) && j.n_eff <= 4 << (sh - 1)) --sh;
    return sh;
  }
  __device__ static void epilogue_pre(const Params& p, const Job& j, SharedTail& sh, const EpiCtx& ec,
                                      EpilogueState& st) {
    st.has_pos = 0;
    if (SPLIT && st.scales_of != j.t1) {
      st.scales_of = j.t1;
      // (from memory four at a time, each waited for, they made half of the warps' time with the loss: steps of three kernels, 1 000 000 x 64
      // at batch 200 500 and 485 us, with the loss 666 and 610, at 512 1 360 and 1 234; 500 000 x 768 at 512 with the loss 1 336 and 1 290)
      const float2 two = *reinterpret_cast<const float2*>(p.x_scale + j.b0 + (ec.h << col_shift(j)) + 2 * ec.lane);
      *reinterpret_cast<float2*>(ec.stage + 8 * ec.lane) = two;
      __syncwarp();
    }
    if (j.a0 >= j.rows) return;                     // second CTA of a pair on a chunk's last tile: no rows
    const int bkt = j.chunk * p.bkt_per_chunk + (j.a0 >> 7);      // buckets are per 128 label rows
    int beg, end;
    if (bkt == st.next_bkt) {
      beg = st.next_beg;
      end = st.next_end;
    } else {
      beg = p.bucket_off[bkt];
      end = p.bucket_off[bkt + 1];
    }
    st.has_pos = end > beg;
    if (!st.has_pos) return;
    constexpr int kWordsPerRow = kTileN / 32;
    const int cs = col_shift(j), word = min(cs, 5);              // log2 of the columns that share a word: of one warp
    __syncwarp();
    for (int w = ec.lane; w < 32 * kWordsPerRow; w += 32) {
      if (((w % kWordsPerRow) << word) >> cs == ec.h) ec.bitmap[ec.q * 32 * kWordsPerRow + w] = 0u;
    }
    __syncwarp();
    for_each_entry<8>(p.bucket_ent, beg, end, ec.lane, [&](uint32_t ent) {
      const int lrow = (int)(ent >> 16), bl = (int)(ent & 0xFFFFu) - j.b0;
      if ((lrow >> 5) == ec.q && bl >= 0 && bl < kTileN && bl >> cs == ec.h)
        atomicOr(&ec.bitmap[lrow * kWordsPerRow + (bl >> word)], 1u << (bl & ((1 << word) - 1)));
    });
    __syncwarp();
  }
  __device__ static void epilogue(const Params& p, const Job& j, uint32_t taddr, bool have_acc,
                                  SharedTail& sh, const EpiCtx& ec, EpilogueState& st) {
    const int row = ec.q * 32 + ec.lane;
    const bool row_valid = j.a0 + row < j.rows;     // the rows that pad a chunk to whole tiles are written as zero
    const int cs = col_shift(j), first = ec.h << cs, c_end = min(j.n_eff, (ec.h + 1) << cs);
    if (SPLIT && LOSS && cs == 4) {
      if (first < c_end) columns<16>(p, j, taddr, have_acc, ec, st, row, row_valid, first, first);
      return;
    }
    for (int c0 = first; c0 < c_end; c0 += 32) columns<32>(p, j, taddr, have_acc, ec, st, row, row_valid, first, c0);
  }
  // COLS neighbouring columns from c0 on, of those from `first` on that the warp has
  template <int COLS>
  __device__ __forceinline__ static void columns(const Params& p, const Job& j, uint32_t taddr, bool have_acc, const EpiCtx& ec, EpilogueState& st,
                                                 int row, bool row_valid, [[maybe_unused]] int first, int c0) {
    const int crow = j.c_row + row;
    uint32_t v[COLS];
    if (have_acc) {
      if constexpr (COLS == 32) tmem_ld32(taddr + c0, v);
      else tmem_ld16(taddr + c0, v);
      tmem_ld_wait();
    } else {
#pragma unroll
      for (int i = 0; i < COLS; ++i) v[i] = 0u;
    }
    const uint32_t bits = st.has_pos ? ec.bitmap[row * (kTileN / 32) + c0 / COLS] : 0u;
    uint32_t out[COLS / 2];
    SoftplusSum sp;
    [[maybe_unused]] uint64_t sc[2] = {0ull, 0ull};
    // Per pair: one packed cvt rounds the logits to bf16, ex2 + rcp give the sigmoid, one packed cvt
    // rounds and packs it.  The two special-function operations per logit are what bounds this epilogue.
    // (Keeping the next column group's accumulator load in flight in a second register buffer was
    // measured: 17 more registers, forward 5 % slower.)
#pragma unroll
    for (int i = 0; i < COLS; i += 2) {
      if (SPLIT && (i & 2) == 0) shared_scales(smem_u32(ec.stage) + 4u * (uint32_t)(c0 - first + i), sc);
      const uint32_t zz = SPLIT ? scaled_bf16x2(v[i], v[i + 1], sc[(i >> 1) & 1])
                                : pack_bf16x2(__uint_as_float(v[i]) * p.w_scale, __uint_as_float(v[i + 1]) * p.w_scale);
      const float z0 = __uint_as_float(zz << 16), z1 = __uint_as_float(zz & 0xFFFF0000u);
      const float s0 = fast_sigmoid(z0), s1 = fast_sigmoid(z1);
      out[i >> 1] = pack_bf16x2(s0, s1);
      if (LOSS) {
        const int left = p.batch - (j.b0 + c0 + i);             // the same for the whole warp
        if (left > 1) sp.add(z0, z1);
        else if (left == 1) sp.add(z0);
      }
    }
    if (LOSS && row_valid) st.loss += sp.value();
    // positives: G = bf16(sigmoid) - 1 in bf16 arithmetic.  Rare (a few thousand pairs per step), so
    // only threads that own one take this path; indices stay compile-time to keep out[] in registers.
    if (bits != 0u) {
#pragma unroll
      for (int i = 0; i < COLS / 2; ++i) {
        const uint32_t two = (bits >> (2 * i)) & 3u;
        if (two == 0u) continue;
        const uint32_t word = out[i];
        float lo = __uint_as_float(word << 16), hi = __uint_as_float(word & 0xFFFF0000u);
        if (two & 1u) lo = bf16_round(lo - 1.0f);
        if (two & 2u) hi = bf16_round(hi - 1.0f);
        out[i] = __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632);
        if (LOSS && row_valid) {
          // loss term -y*z: z recomputed from the accumulator with the same rounding
          float2 two_sc = make_float2(p.w_scale, p.w_scale);
          if constexpr (SPLIT) two_sc = reinterpret_cast<const float2*>(ec.stage)[(c0 - first) / 2 + i];
          if ((two & 1u) && j.b0 + c0 + 2 * i < p.batch) st.loss -= bf16_round(__uint_as_float(v[2 * i]) * two_sc.x);
          if ((two & 2u) && j.b0 + c0 + 2 * i + 1 < p.batch) st.loss -= bf16_round(__uint_as_float(v[2 * i + 1]) * two_sc.y);
        }
      }
    }
    // rows beyond the chunk and batch columns beyond the batch carry G = 0
    if (!row_valid) {
#pragma unroll
      for (int i = 0; i < COLS / 2; ++i) out[i] = 0u;
    } else if (j.b0 + c0 + COLS > p.batch) {
#pragma unroll
      for (int i = 0; i < COLS / 2; ++i) {
        const int b = j.b0 + c0 + 2 * i;
        if (b >= p.batch) out[i] = 0u;
        else if (b + 1 >= p.batch) out[i] &= 0x0000FFFFu;
      }
    }
    if constexpr (WRITE_G8) {
      // the same 32 values once more as e4m3(G * 256): one 32-byte sector
      if (j.b0 + c0 < p.bpad) {
        U32x8 g8;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t w0 = out[2 * k], w1 = out[2 * k + 1];
          const uint32_t lo = float2_to_e4m3x2(__uint_as_float(w0 << 16) * kG8Scale, __uint_as_float(w0 & 0xFFFF0000u) * kG8Scale);
          const uint32_t hi = float2_to_e4m3x2(__uint_as_float(w1 << 16) * kG8Scale, __uint_as_float(w1 & 0xFFFF0000u) * kG8Scale);
          g8.v[k] = lo | (hi << 16);
        }
        st_global_256(p.G8 + (size_t)crow * p.bpad + j.b0 + c0, g8);
      }
    }
    if constexpr (kTmaG) {
      const int part = (c0 >> 5) & 1;
      if (part == 0) {
        if (ec.lane == 0) bulk_wait_read_all();        // the box has been read by its last store
        __syncwarp();
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<uint4*>(ec.stage + ec.lane * 128 + (((4 * part + i) ^ (ec.lane & 7)) << 4)) =
            make_uint4(out[4 * i], out[4 * i + 1], out[4 * i + 2], out[4 * i + 3]);
      if (part == 1) {
        fence_proxy_async();
        __syncwarp();
        if (ec.lane == 0) {
          tma_store_2d(ec.map_c, smem_u32(ec.stage), j.b0 + c0 - 32, j.c_row + ec.q * 32);
          bulk_commit_group();
        }
      }
    } else {
      // two 256-bit stores: every thread writes whole 32-byte sectors of its row
      __nv_bfloat16* grow = p.G + (size_t)crow * p.bpad + j.b0 + c0;
#pragma unroll
      for (int i = 0; i < COLS / 16; ++i) {
        if (j.b0 + c0 + 16 * i < p.bpad) {
          U32x8 o8;
#pragma unroll
          for (int k = 0; k < 8; ++k) o8.v[k] = out[8 * i + k];
          st_global_256(grow + 16 * i, o8);
        }
      }
    }
  }
  __device__ static void epilogue_end(const Params& p, SharedTail&, const EpiCtx& ec, EpilogueState& st) {
    if constexpr (kTmaG) {
      if (ec.lane == 0) bulk_wait_all();
      __syncwarp();
    }
    if (!LOSS) return;
    float v = st.loss;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (ec.lane == 0 && p.loss_partial != nullptr) p.loss_partial[blockIdx.x * kEpiWarps + ec.slot] = (double)v;
  }
};

// -------------------------------------------------------------------------------------------------
// Fused dW + SGD update (reference: fuse_kernel.py:63-131 naive_matmul_k / matmul_update; for bf16
// weights chunked.py:119 + stochastic_rounding_kernel.py:65-99).
// -------------------------------------------------------------------------------------------------
struct UpdParams {
  LabelTiles lt;
  const CUtensorMap* w_maps;   // one per chunk, in device memory: boxes of 128 rows x 128 bytes
  int n_dtiles;
  FastDiv div_dtiles;      // of n_dtiles
  int d;
  int k_steps;             // cdiv(bpad, 64)
  float lr_eff;            // lr / w_scale
  float wd;
  unsigned long long seed, step;
  uint32_t rkey[kSrRounds][2];   // Philox round keys (seed + round * Weyl constants), filled on the host: they sit in
                              // the constant bank, so a round costs two multiplies and two 3-input xors
  uint32_t sr_x1, sr_y1, sr_z1;  // step-dependent parts of the first two rounds (see philox_prepare)
  unsigned long long elem0;   // global flat element index of the handle's W[0][0] (Philox counter origin)
  int round_dw_bf16;
  // Kahan-compensated head rows (reference: fuse_kernel.py:202-287, chunked_head_kahan_fp8xmc_clf.py:127-131)
  void* kahan;             // compensation buffer, [kahan_rows x d] bf16 or e5m2; or nullptr
  int kahan_rows;          // rows [0, kahan_rows) of chunk 0 are compensated
  int kahan_e5m2;
  int* status;
};

// OPS8: the dW contraction takes e4m3 operands (G * 256 and X, both as the forward already quantises
// them) instead of bf16 ones; the caller folds the 1/256 into lr_eff.  Off in every reference-parity path.
template <bool W8, bool SR, bool ROUND_DW, bool HAS_WD, bool KAHAN = false, bool OPS8 = false>
struct UpdPolicy {
  using Params = UpdParams;
  static constexpr bool kMnMajor = false;
  static constexpr bool kChunkMaps = true;   // Params::w_maps are the maps of one operand or of the epilogue's tile
  static constexpr bool kFp8 = OPS8;
  static constexpr uint32_t kFmt = OPS8 ? 0u : 1u;
  static constexpr int kElemsPerRow = OPS8 ? 128 : 64;
  static constexpr int kEpiWarps = 16;
  // The tile's 128 x 256 weights come in by TMA while the main loop runs and go back by TMA, through 32 KB slots
  // paid for with operand stages (e4m3 with a single slot: the refill has to wait for the previous tile's store
  // and the pipeline serialises, 30 % slower).  bf16 weights pass in two parts of 128 columns through
  // three slots, which leaves four operand stages: whole 64 KB tiles in two slots left three, 3 % slower
  // at batch 1024.  (Read and written by the epilogue threads as 32-byte pieces of 32 different rows, with
  // nothing requested ahead, the bf16 update of 131 072 x 768 at batch 256 took 215 us; now 100.)
  static constexpr bool kCTile = true;
  static constexpr int kCBufs = W8 ? 2 : 3;
  static constexpr int kCParts = W8 ? 1 : 2;
  static constexpr int kSplit = 0, kXRows = 0;
  __device__ static int x_rows(const Params&) { return 0; }
  static constexpr bool kConv = false, kEarlyWeights = false;
  static constexpr bool kBitmap = false;
  static constexpr int kEpiStage = 0;
  static constexpr int kWaitRoles = kRoleAll;
  __device__ static bool wait_all(const Params&) { return true; }
  __device__ static long long wait_limit(const Params&) { return kWaitLimitCycles; }
  __device__ static bool skip_load(const Params&, int, int) { return false; }
  static constexpr int kStages = W8 ? 3 : 2;
  static constexpr int kStagesPair = W8 ? 5 : 4;
  // the weight block: columns [c_col, c_col + 256) of the CTA's 128 rows; not stored back when the CTA's
  // rows lie wholly beyond the chunk (second CTA of a pair on an odd last tile)
  __device__ static int c_col(const Job& j) { return j.b0; }
  __device__ static bool c_store(const Params&, const Job& j) { return j.c_row < j.rows; }
  __device__ static const CUtensorMap* map_a(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_b(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_c(const Params& p, const Job& j, const CUtensorMap*) { return p.w_maps + j.chunk; }
  static constexpr int kGroups = ((kTileN / 32) + (kEpiWarps / 4) - 1) / (kEpiWarps / 4);   // 32-column groups per thread and tile
  using EpilogueState = NoState;

  __device__ static int num_tiles(const Params& p) { return p.lt.count * p.n_dtiles; }
  __device__ static void job(const Params& p, int tile, Job& j) {
    j.t0 = fast_div(tile, p.div_dtiles);
    j.t1 = tile - j.t0 * p.n_dtiles;
    j.a0 = j.t0 * p.lt.m_rows;           // rows of G
    p.lt.locate(j.t0, j, j.c_row);       // rows of the chunk
    j.b0 = j.t1 * kTileN;     // rows of X^T = feature index
    j.k_begin = 0;
    j.k_steps = p.k_steps;
    j.n_eff = min(kTileN, round_up16(p.d - j.b0));
  }
  __device__ static void epilogue_begin(const Params&, EpilogueState&) {}
  __device__ static void epilogue_end(const Params&, SharedTail&, const EpiCtx&, EpilogueState&) {}

  __device__ static void epilogue_pre(const Params&, const Job&, SharedTail&, const EpiCtx&, EpilogueState&) {}
  __device__ static void epilogue_prefetch(const Params&, const Job&, EpilogueState&) {}
  __device__ static float new_weight(const Params& p, float w, uint32_t acc_bits) {
    // no run-time branches in here: they would cut the per-element code into tiny basic blocks
    float a = __uint_as_float(acc_bits);
    if constexpr (ROUND_DW) a = bf16_round(a);
    if constexpr (HAS_WD) a = fmaf(p.wd, w, a);
    return fmaf(-p.lr_eff, a, w);
  }
  // the same for two neighbouring elements, two at a time where the hardware has packed forms
  __device__ static uint64_t new_weight2(const Params& p, float w0, float w1, uint32_t acc0, uint32_t acc1) {
    uint64_t a;
    if constexpr (ROUND_DW) {
      const uint32_t r = pack_bf16x2(__uint_as_float(acc0), __uint_as_float(acc1));
      a = pack_f32x2(__uint_as_float(r << 16), __uint_as_float(r & 0xFFFF0000u));
    } else {
      a = pack_f32x2(__uint_as_float(acc0), __uint_as_float(acc1));
    }
    const uint64_t w = pack_f32x2(w0, w1);
    if constexpr (HAS_WD) a = fma_f32x2(pack_f32x2(p.wd, p.wd), w, a);
    return fma_f32x2(pack_f32x2(-p.lr_eff, -p.lr_eff), a, w);
  }

  // ------------------------------------------------------------------------------------------------
  // Philox4x32, counter (q_lo, q_hi, step_lo, step_hi).  Two of the counter's words never change within a
  // launch and q_hi only every 2^35 elements, so one multiply of each of the first two rounds and
  // what it feeds are the same for all elements of a row: PhiloxRow holds them (two multiplies and one
  // xor fewer per call of seven rounds).
  // ------------------------------------------------------------------------------------------------
  static constexpr uint32_t kM0 = 0xD2511F53u, kM1 = 0xCD9E8D57u;
  struct PhiloxRow {
    uint32_t q_hi, z2, w2, z3;
  };
  __device__ static void philox_row(const Params& p, uint32_t q_hi, PhiloxRow& pr) {
    pr.q_hi = q_hi;
    const unsigned long long m = (unsigned long long)kM0 * (p.sr_x1 ^ q_hi);
    pr.z2 = (uint32_t)(m >> 32) ^ p.rkey[1][1];
    pr.w2 = (uint32_t)m;
    pr.z3 = pr.w2 ^ p.rkey[2][1];
  }
  __device__ static uint4 philox(const Params& p, const PhiloxRow& pr, uint32_t q_lo) {
    const unsigned long long a1 = (unsigned long long)kM0 * q_lo;                              // round 1
    const unsigned long long b2 = (unsigned long long)kM1 * ((uint32_t)(a1 >> 32) ^ p.sr_z1);  // round 2
    const unsigned long long a3 = (unsigned long long)kM0 * ((uint32_t)(b2 >> 32) ^ p.sr_y1);  // round 3
    const unsigned long long b3 = (unsigned long long)kM1 * ((uint32_t)a1 ^ pr.z2);
    uint4 c = make_uint4((uint32_t)(b3 >> 32) ^ (uint32_t)b2 ^ p.rkey[2][0], (uint32_t)b3, (uint32_t)(a3 >> 32) ^ pr.z3,
                         (uint32_t)a3);
#pragma unroll
    for (int rd = 3; rd < kSrRounds; ++rd) {
      const unsigned long long p0 = (unsigned long long)kM0 * c.x;
      const unsigned long long p1 = (unsigned long long)kM1 * c.z;
      c = make_uint4((uint32_t)(p1 >> 32) ^ c.y ^ p.rkey[rd][0], (uint32_t)p1, (uint32_t)(p0 >> 32) ^ c.w ^ p.rkey[rd][1],
                     (uint32_t)p0);
    }
    return c;
  }

  // ------------------------------------------------------------------------------------------------
  // e4m3 weights, four consecutive elements of one row.
  //
  // With stochastic rounding this is what bounds the kernel when the batch is small.  Per scheduler and
  // element (of a warp) the multiplier-add pipe is busy for 6 cycles with the 12 wide multiplies that eight
  // elements share (4 cycles each), 3 with the three packed fp32 operations (2 cycles each for two elements) and 2
  // with the rounding add, while the other integer pipe (2 cycles an instruction) has the conversions
  // and the xors; 16 cycles in all (20 with half-word extraction by
  // mask and shift and a running sum as the non-finite test, 16.2 with a mask for what lies below the grid).
  //   - the rounding bits are added by a 16-bit dot product with weights (16, 0) or (0, 16): one
  //     instruction instead of extract and shift-add;
  //   - what lies below the grid is cut off by the conversion itself (four elements, towards zero), where a mask
  //     took an instruction per element, and weights are widened by the mixed-precision multiply-add: same bits,
  //     one-kernel step of 4 001 x 768 batch 16 19.76 -> 19.63 us, step of 131 072 x 768 batch 256 208.0 -> 206.0;
  //   - non-finite updates (the bare add-and-mask would mangle a NaN pattern) show in a running three-input
  //     maximum of magnitudes, half an instruction per element; the caller looks at it once per sixteen and
  //     redoes them with update8_careful.
  // old: the four weights as they were, as bf16 (two words; unused outputs cost nothing).
  __device__ static uint32_t update4(const Params& p, const uint32_t* v, uint32_t w, uint32_t r0, uint32_t r1, float& mx,
                                     uint32_t* old) {
    float f[4];
    e4m3x4_to_float4<SR>(w, f);
    old[0] = pack_bf16x2(f[0], f[1]);
    old[1] = pack_bf16x2(f[2], f[3]);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      uint64_t o = new_weight2(p, f[i], f[i + 1], v[i], v[i + 1]);
      if (SR) {
        // both elements of a pair draw from the same Philox word: element j takes half (j & 1) of word j >> 1
        const uint32_t w32 = i ? r1 : r0;
        float x0, x1;
        unpack_f32x2(mul_f32x2(o, pack_f32x2(kSrDown, kSrDown)), x0, x1);
        mx = max3_abs_nan(mx, x0, x1);
        const uint32_t b0 = add_low16x16(__float_as_uint(x0), w32);
        const uint32_t b1 = add_high16x16(__float_as_uint(x1), w32);
        o = mul_f32x2(pack_f32x2(__uint_as_float(b0), __uint_as_float(b1)), pack_f32x2(kSrUp, kSrUp));
      }
      unpack_f32x2(o, f[i], f[i + 1]);
    }
    return SR ? float4_to_e4m3x4_rz(f[0], f[1], f[2], f[3]) : float4_to_e4m3x4(f[0], f[1], f[2], f[3]);
  }
  // sixteen consecutive elements: accumulators va, vb, weights w, two Philox results
  __device__ static uint4 update16(const Params& p, const uint32_t (&va)[8], const uint32_t (&vb)[8], uint4 w, uint4 ra, uint4 rb,
                                   uint32_t (&old)[8]) {
    float mx = 0.f;                                      // finite updates stay below 2^8 after scaling
    uint4 o;
    o.x = update4(p, va, w.x, ra.x, ra.y, mx, old);
    o.y = update4(p, va + 4, w.y, ra.z, ra.w, mx, old + 2);
    o.z = update4(p, vb, w.z, rb.x, rb.y, mx, old + 4);
    o.w = update4(p, vb + 4, w.w, rb.z, rb.w, mx, old + 6);
    if (SR && !(mx < 1.0e30f)) {
      const uint2 oa = update8_careful(p, va[0], va[1], va[2], va[3], va[4], va[5], va[6], va[7], make_uint2(w.x, w.y), ra);
      const uint2 ob = update8_careful(p, vb[0], vb[1], vb[2], vb[3], vb[4], vb[5], vb[6], vb[7], make_uint2(w.z, w.w), rb);
      o = make_uint4(oa.x, oa.y, ob.x, ob.y);
    }
    return o;
  }

  // Eight elements one by one with the NaN-preserving rounding (rare).
  __device__ __noinline__ static uint2 update8_careful(const Params& p, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3,
                                                       uint32_t v4, uint32_t v5, uint32_t v6, uint32_t v7, uint2 wraw, uint4 r) {
    const uint32_t v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
    const uint32_t rw[2] = {wraw.x, wraw.y};
    const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
    uint32_t ow[2] = {0u, 0u};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float w = e4m3x2_to_float2((uint16_t)(rw[e >> 2] >> (8 * (e & 3)))).x;
      const uint32_t r16 = (e & 1) ? (rr[e >> 1] >> 16) : (rr[e >> 1] & 0xFFFFu);
      const float o = sr_e4m3(new_weight(p, w, v[e]), r16);
      ow[e >> 2] |= ((uint32_t)float2_to_e4m3x2(o, 0.f) & 0xFFu) << (8 * (e & 3));
    }
    return make_uint2(ow[0], ow[1]);
  }

  // Kahan-compensated rows: w = W + D - lr*acc; W' = round(w); D' = cast(D + W - W' - lr*acc)
  // (fuse_kernel.py:253-273).  Sixteen consecutive elements, d their D, two at a time as update16; false,
  // and nothing changed, where an update is not finite (e5m2 terms: where D' is beyond their largest, too, as this
  // conversion saturates).  Eight elements one by one, update8_kahan, take three times the instructions, and came on top
  // of update16: tiles of compensated rows 30 us where others took 10.  One-kernel step of 312 330 x 768, batch 128, a tenth of
  // the rows compensated in bf16 402 -> 370 us; 312 330 x 768, batch 256 (the update kernel) 470 -> 390, 20 of them by other
  // kernels' gains.  With e5m2 terms 700 000 x 768, batch 64 882 -> 604 (left to update8_kahan in kernels made for sixteen at
  // a time 960), batch 200 1344 -> 868.
  template <bool E5M2>
  __device__ static bool update16_kahan(const Params& p, const uint32_t (&va)[8], const uint32_t (&vb)[8], uint4 w, uint4 ra, uint4 rb,
                                        uint4 (&d)[2], uint4& out) {
    const uint32_t ww[4] = {w.x, w.y, w.z, w.w}, rr[8] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y, rb.z, rb.w};
    uint32_t dd[8] = {d[0].x, d[0].y, d[0].z, d[0].w, d[1].x, d[1].y, d[1].z, d[1].w}, oo[4];     // e5m2: four to a word
    const uint64_t lr = pack_f32x2(p.lr_eff, p.lr_eff), nlr = pack_f32x2(-p.lr_eff, -p.lr_eff), minus = pack_f32x2(-1.f, -1.f);
    float mx = 0.f, md = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g) {                         // four elements: one word of W
      const uint32_t* v = g < 2 ? va + 4 * g : vb + 4 * (g - 2);
      float f[4], n[4], df[4];
      e4m3x4_to_float4<SR>(ww[g], f);
      if constexpr (E5M2) {
        e5m2x4_to_float4(dd[g], df);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) df[i] = __uint_as_float(i & 1 ? dd[2 * g + (i >> 1)] & 0xFFFF0000u : dd[2 * g + (i >> 1)] << 16);
      }
      uint64_t a[2], s[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint32_t w32 = rr[2 * g + i];
        a[i] = pack_f32x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        s[i] = add_f32x2(pack_f32x2(f[2 * i], f[2 * i + 1]), pack_f32x2(df[2 * i], df[2 * i + 1]));
        uint64_t o = fma_f32x2(nlr, a[i], s[i]);
        if (SR) {
          float x0, x1;
          unpack_f32x2(mul_f32x2(o, pack_f32x2(kSrDown, kSrDown)), x0, x1);
          mx = max3_abs_nan(mx, x0, x1);
          o = mul_f32x2(pack_f32x2(__uint_as_float(add_low16x16(__float_as_uint(x0), w32)), __uint_as_float(add_high16x16(__float_as_uint(x1), w32))),
                        pack_f32x2(kSrUp, kSrUp));
        }
        unpack_f32x2(o, n[2 * i], n[2 * i + 1]);
      }
      oo[g] = SR ? float4_to_e4m3x4_rz(n[0], n[1], n[2], n[3]) : float4_to_e4m3x4(n[0], n[1], n[2], n[3]);
      e4m3x4_to_float4<SR>(oo[g], n);                         // the value W' holds
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint64_t rest = fma_f32x2(minus, pack_f32x2(n[2 * i], n[2 * i + 1]), s[i]);
        unpack_f32x2(fma_f32x2(minus, mul_f32x2(lr, a[i]), rest), df[2 * i], df[2 * i + 1]);
      }
      if constexpr (E5M2) {
        md = max3_abs_nan(max3_abs_nan(md, df[0], df[1]), df[2], df[3]);
        dd[g] = float4_to_e5m2x4(df[0], df[1], df[2], df[3]);
      } else {
        dd[2 * g] = pack_bf16x2(df[0], df[1]);
        dd[2 * g + 1] = pack_bf16x2(df[2], df[3]);
      }
    }
    if ((SR && !(mx < 1.0e30f)) || (E5M2 && !(md <= kE5m2Max))) return false;
    out = make_uint4(oo[0], oo[1], oo[2], oo[3]);
    d[0] = make_uint4(dd[0], dd[1], dd[2], dd[3]);
    if constexpr (!E5M2) d[1] = make_uint4(dd[4], dd[5], dd[6], dd[7]);
    return true;
  }

  // The same, eight elements one by one: what is not finite, or beyond e5m2.
  __device__ __noinline__ static uint2 update8_kahan(const Params& p, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3,
                                                     uint32_t v4, uint32_t v5, uint32_t v6, uint32_t v7, uint2 wraw, uint4 r,
                                                     void* krow) {
    const uint32_t v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
    const uint32_t rw[2] = {wraw.x, wraw.y};
    const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
    float dv[8];
    if (p.kahan_e5m2) {
      const uint2 raw = *reinterpret_cast<const uint2*>(krow);
      const uint32_t rk[2] = {raw.x, raw.y};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(rk[i >> 1] >> (16 * (i & 1))), __NV_E5M2);
        const float2 f = __half22float2(*reinterpret_cast<__half2*>(&hr));
        dv[2 * i] = f.x; dv[2 * i + 1] = f.y;
      }
    } else {
      const uint4 raw = *reinterpret_cast<const uint4*>(krow);
      const uint32_t rk[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        dv[2 * i] = bf16_bits_to_float(rk[i] & 0xFFFFu);
        dv[2 * i + 1] = bf16_bits_to_float(rk[i] >> 16);
      }
    }
    uint32_t ow[2] = {0u, 0u};
    float dn[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float wv = e4m3x2_to_float2((uint16_t)(rw[e >> 2] >> (8 * (e & 3)))).x;
      const float a = __uint_as_float(v[e]);
      float o = fmaf(-p.lr_eff, a, __fadd_rn(wv, dv[e]));
      if (SR) o = sr_e4m3(o, (e & 1) ? (rr[e >> 1] >> 16) : (rr[e >> 1] & 0xFFFFu));
      const uint32_t byte = (uint32_t)float2_to_e4m3x2(o, 0.f) & 0xFFu;
      o = e4m3x2_to_float2((uint16_t)byte).x;                       // the value W' holds
      ow[e >> 2] |= byte << (8 * (e & 3));
      dn[e] = __fsub_rn(__fsub_rn(__fadd_rn(dv[e], wv), o), __fmul_rn(p.lr_eff, a));
    }
    if (p.kahan_e5m2) {
      uint32_t ok[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t pr = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(dn[2 * i], dn[2 * i + 1]), __NV_NOSAT, __NV_E5M2);
        if (i & 1) ok[i >> 1] |= pr << 16; else ok[i >> 1] = pr;
      }
      *reinterpret_cast<uint2*>(krow) = make_uint2(ok[0], ok[1]);
    } else {
      *reinterpret_cast<uint4*>(krow) = make_uint4(pack_bf16x2(dn[0], dn[1]), pack_bf16x2(dn[2], dn[3]),
                                                   pack_bf16x2(dn[4], dn[5]), pack_bf16x2(dn[6], dn[7]));
    }
    return make_uint2(ow[0], ow[1]);
  }

  // Sixteen elements of a compensated row, the first of them element `at` of the buffer (a multiple of 16: rows are multiples
  // of 64 elements).  Their terms are asked for ahead (kahan_fetch), before the random bits are drawn: they come from
  // memory, 32 or 16 bytes a row.
  template <bool E5M2>
  __device__ static void kahan_fetch(const Params& p, size_t at, uint4 (&d)[2]) {
    const uint4* krow = reinterpret_cast<const uint4*>(reinterpret_cast<uint8_t*>(p.kahan) + (E5M2 ? at : 2 * at));
    d[0] = krow[0];
    if constexpr (!E5M2) d[1] = krow[1];
  }
  template <bool E5M2>
  __device__ static uint4 kahan16(const Params& p, const uint32_t (&va)[8], const uint32_t (&vb)[8], uint4 w, uint4 ra, uint4 rb, size_t at,
                                  uint4 (&d)[2]) {
    uint8_t* krow = reinterpret_cast<uint8_t*>(p.kahan) + (E5M2 ? at : 2 * at);
    uint4 out;
    if (update16_kahan<E5M2>(p, va, vb, w, ra, rb, d, out)) {
      reinterpret_cast<uint4*>(krow)[0] = d[0];
      if constexpr (!E5M2) reinterpret_cast<uint4*>(krow)[1] = d[1];
      return out;
    }
    const uint2 oa = update8_kahan(p, va[0], va[1], va[2], va[3], va[4], va[5], va[6], va[7], make_uint2(w.x, w.y), ra, krow);
    const uint2 ob = update8_kahan(p, vb[0], vb[1], vb[2], vb[3], vb[4], vb[5], vb[6], vb[7], make_uint2(w.z, w.w), rb, krow + (E5M2 ? 8 : 16));
    return make_uint4(oa.x, oa.y, ob.x, ob.y);
  }

  // the whole tile for e4m3 weights: 2 * kGroups sub-blocks of 16 columns per thread.  The two halves of
  // a sub-block (8 columns, one Philox call each) are independent chains in one basic block: a warp has
  // two of the long multiply-xor chains to interleave, which is what lets four warps per scheduler fill
  // its issue slots.
  __device__ static void epilogue_w8(const Params& p, const Job& j, uint32_t taddr, bool have_acc, const EpiCtx& ec) {
    const int row = ec.q * 32 + ec.lane;
    const int crow = j.c_row + row;
    const bool row_valid = crow < j.rows;
    const unsigned long long erow = p.elem0 + (unsigned long long)p.lt.row_of(j, crow) * p.d + j.b0;
    PhiloxRow pr;
    if (SR) philox_row(p, (uint32_t)(erow >> 35), pr);
#pragma unroll 1
    for (int sb = 0; sb < 2 * kGroups; ++sb) {
      const int c0 = 32 * (ec.h + ec.nsplit * (sb >> 1)) + 16 * (sb & 1);
      if (c0 >= j.n_eff) break;                          // warp-uniform
      // tcgen05.ld / wait::ld are warp-wide (.sync.aligned): issued by all 32 lanes, outside every
      // lane-dependent branch; the loads are asynchronous, so the random bits are drawn while they fly
      uint32_t va[8], vb[8];
      if (have_acc) {
        tmem_ld8(taddr + c0, va);
        tmem_ld8(taddr + c0 + 8, vb);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) va[i] = vb[i] = 0u;
      }
      // 16 weight bytes: one 16-byte piece of the swizzled block
      uint4* wslot = ctile_ptr16(ec.ctile, row, c0);
      const uint4 wraw = *wslot;                         // rows / columns outside the tensor were zero-filled
      bool kahan_row = false;
      uint4 comp[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
      if constexpr (KAHAN) {
        kahan_row = j.chunk == 0 && crow < p.kahan_rows && j.b0 + c0 < p.d;    // (d is a multiple of 16: the sixteen are there or none of them)
        if (kahan_row && row_valid) {
          const size_t at = (size_t)crow * p.d + j.b0 + c0;
          if (p.kahan_e5m2) kahan_fetch<true>(p, at, comp);
          else kahan_fetch<false>(p, at, comp);
        }
      }
      uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
      if (SR) {
        const unsigned long long q = (erow + c0) >> 3;   // even: rows and column groups start at multiples of 16
        if ((uint32_t)(q >> 32) != pr.q_hi) philox_row(p, (uint32_t)(q >> 32), pr);
        ra = philox(p, pr, (uint32_t)q);
        rb = philox(p, pr, (uint32_t)q + 1u);
      }
      if (have_acc) tmem_ld_wait_for(va, vb);
      uint4 out = wraw;
      if (kahan_row) {
        const size_t at = (size_t)crow * p.d + j.b0 + c0;
        if (row_valid) out = p.kahan_e5m2 ? kahan16<true>(p, va, vb, wraw, ra, rb, at, comp) : kahan16<false>(p, va, vb, wraw, ra, rb, at, comp);
      } else {
        uint32_t old[8];
        out = update16(p, va, vb, wraw, ra, rb, old);
      }
      if (row_valid) *wslot = out;                       // in place; the engine stores the block back with TMA
    }
  }

  // bf16 weights, two consecutive elements (one word): stochastic rounding adds the element's 16 random bits
  // below the kept mantissa and truncates (fuse_kernel.py:10-17).  The hardware's conversion gives the same bits for all numbers,
  // infinities among them and what rounds up past the largest, which becomes one.  Something that is not a number it keeps, where
  // the addition runs over into the sign and leaves -0.
  __device__ static uint32_t update2_bf16(const Params& p, uint32_t v0, uint32_t v1, uint32_t w, uint32_t w32) {
    const uint64_t o = new_weight2(p, __uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u), v0, v1);
    float o0, o1;
    unpack_f32x2(o, o0, o1);
    if (SR) return float2_to_bf16x2_rs(o0, o1, w32);
    return pack_bf16x2(o0, o1);
  }
  // the tile's part (128 columns) for bf16 weights, 16 columns at a time as above
  __device__ static void epilogue_bf16(const Params& p, const Job& j, uint32_t taddr, bool have_acc, const EpiCtx& ec) {
    const int row = ec.q * 32 + ec.lane;
    const unsigned long long erow = p.elem0 + (unsigned long long)p.lt.row_of(j, j.c_row + row) * p.d + j.b0;
    PhiloxRow pr;
    if (SR) philox_row(p, (uint32_t)(erow >> 35), pr);
#pragma unroll 1
    for (int sb = 0; sb < 2; ++sb) {
      const int cp = 32 * ec.h + 16 * sb, c0 = 128 * ec.part + cp;    // column within the part, within the tile
      if (c0 >= j.n_eff) break;                          // warp-uniform
      uint32_t va[8], vb[8];
      if (have_acc) {
        tmem_ld8(taddr + c0, va);
        tmem_ld8(taddr + c0 + 8, vb);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) va[i] = vb[i] = 0u;
      }
      uint4* slot_a = ctile_ptr16(ec.ctile, row, 2 * cp);
      uint4* slot_b = ctile_ptr16(ec.ctile, row, 2 * cp + 16);
      const uint4 wa = *slot_a, wb = *slot_b;            // rows / columns outside the tensor were zero-filled
      uint4 ra = make_uint4(0u, 0u, 0u, 0u), rb = ra;
      if (SR) {
        const unsigned long long q = (erow + c0) >> 3;
        if ((uint32_t)(q >> 32) != pr.q_hi) philox_row(p, (uint32_t)(q >> 32), pr);
        ra = philox(p, pr, (uint32_t)q);
        rb = philox(p, pr, (uint32_t)q + 1u);
      }
      if (have_acc) tmem_ld_wait_for(va, vb);
      *slot_a = make_uint4(update2_bf16(p, va[0], va[1], wa.x, ra.x), update2_bf16(p, va[2], va[3], wa.y, ra.y),
                           update2_bf16(p, va[4], va[5], wa.z, ra.z), update2_bf16(p, va[6], va[7], wa.w, ra.w));
      *slot_b = make_uint4(update2_bf16(p, vb[0], vb[1], wb.x, rb.x), update2_bf16(p, vb[2], vb[3], wb.y, rb.y),
                           update2_bf16(p, vb[4], vb[5], wb.z, rb.z), update2_bf16(p, vb[6], vb[7], wb.w, rb.w));
    }
  }

  __device__ static void epilogue(const Params& p, const Job& j, uint32_t taddr, bool have_acc,
                                  SharedTail&, const EpiCtx& ec, EpilogueState&) {
    if (j.c_row >= j.rows) return;                  // whole CTA tile beyond the chunk (pairs only)
    if constexpr (W8) epilogue_w8(p, j, taddr, have_acc, ec);
    else epilogue_bf16(p, j, taddr, have_acc, ec);
  }
};

// -------------------------------------------------------------------------------------------------
// Inference logits (reference: chunked.py:48-53, chunked_fp8xmc_clf.py:45-60 xfc_forward):
// out[b][col0 + r] = bf16(w_scale * <x[b], W[r]>).  Batch rows sit on the TMEM lanes so that a thread
// stores runs of consecutive labels.
// -------------------------------------------------------------------------------------------------
struct LogitsParams {
  int m_rows;              // batch rows per M tile: 128, or 256 on CTA pairs
  int batch;
  int n_mtiles;            // batch tiles of m_rows
  FastDiv div_mtiles;      // of n_mtiles
  LabelTiles lt;           // label tiles of 256
  const CUtensorMap* w_maps;   // one per chunk, in device memory
  int k_steps;
  int own_prep;            // the kernel before this one is this call's preparation of X
  int x_rows;              // rows of a box of X
  float w_scale;
  const float* x_scale;    // split embeddings: see FwdParams
  int part_rows;
  const uint8_t* x_wide;
  __nv_bfloat16* out;      // [batch x ld_out]
  long long ld_out;
  long long n_out;         // columns >= n_out are not written
  int* status;
};

template <bool FP8, Simulated SIM = kSimNone>
struct LogitsPolicy {
  static constexpr bool SPLIT = SIM == kSimSplit;
  static_assert(SIM == kSimNone || FP8 == SPLIT, "the parts are FP8 operands, the converted weights bf16");
  using Params = LogitsParams;
  static constexpr bool kMnMajor = false;
  static constexpr bool kChunkMaps = true;   // Params::w_maps are the maps of one operand or of the epilogue's tile
  static constexpr bool kFp8 = FP8;
  static constexpr uint32_t kFmt = FP8 ? 0u : 1u;
  static constexpr int kElemsPerRow = FP8 ? 128 : 64;
  static constexpr int kEpiWarps = 8;
  static constexpr int kStages = 3;
  static constexpr int kStagesPair = SIM != kSimNone ? 4 : 5;
  static constexpr int kSplit = SPLIT ? 1 : 0, kXRows = 1;
  __device__ static int x_rows(const Params& p) { return p.x_rows; }
  __device__ static int tile_rows(const Params& p) { return p.m_rows; }
  __device__ static int x_tile(const Job& j) { return j.t0; }
  static constexpr bool kConv = SIM == kSimConvert, kEarlyWeights = !kConv;
  static constexpr bool kCTile = false;
  static constexpr int kCBufs = 1;
  static constexpr int kCParts = 1;
  static constexpr bool kBitmap = false;
  static constexpr int kEpiBoxes = SIM != kSimNone ? 1 : 2;      // boxes of 32 rows x 64 columns
  static constexpr int kEpiStage = 4096 * kEpiBoxes;
  // the kernel before this one, or the caller's, wrote X
  static constexpr int kWaitRoles = kRoleAll;
  __device__ static bool wait_all(const Params&) { return true; }
  __device__ static long long wait_limit(const Params&) { return kWaitLimitCycles; }
  __device__ static bool skip_load(const Params&, int, int) { return false; }
  struct EpilogueState {
    uint32_t boxes;        // boxes stored so far
  };
  __device__ static const CUtensorMap* map_a(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_b(const Params& p, const Job& j, const CUtensorMap*) { return p.w_maps + j.chunk; }
  __device__ static const CUtensorMap* map_c(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static int num_tiles(const Params& p) { return p.n_mtiles * p.lt.count; }
  __device__ static void job(const Params& p, int tile, Job& j) {
    j.t1 = fast_div(tile, p.div_mtiles);   // label tile (adjacent CTAs share it)
    j.t0 = tile - j.t1 * p.n_mtiles;       // batch tile
    j.a0 = j.t0 * p.m_rows;
    j.c_row = j.a0;
    p.lt.locate(j.t1, j, j.b0);
    j.k_begin = 0;
    j.k_steps = p.k_steps;
    j.n_eff = min(kTileN, round_up16(j.rows - j.b0));
  }
  __device__ static void epilogue_begin(const Params&, EpilogueState& st) { st.boxes = 0u; }
  __device__ static void epilogue_pre(const Params&, const Job&, SharedTail&, const EpiCtx&, EpilogueState&) {}
  __device__ static void epilogue_prefetch(const Params&, const Job&, EpilogueState&) {}
  __device__ static void epilogue_end(const Params&, SharedTail&, const EpiCtx& ec, EpilogueState&) {
    if (ec.lane == 0) bulk_wait_all();
    __syncwarp();
  }
  // A warp takes 128 columns of its 32 rows in two boxes of 64, which go through shared memory and out by TMA: whole
  // 128-byte lines.  What bounds the kernel is the output (2 bytes per logit against 1 or 2 of weights per feature
  // row): stored by the threads, 64 bytes of 32 rows at a time, 300 000 x 768, batch 512 took 166 us, 3.2 TB/s.
  // Columns that TMA may not write -- beyond the chunk or n_out, or at an address that is not a multiple of 16
  // bytes -- are stored by the threads.
  __device__ static void epilogue(const Params& p, const Job& j, uint32_t taddr, bool have_acc,
                                  SharedTail&, const EpiCtx& ec, EpilogueState& st) {
    if (j.a0 + ec.q * 32 >= p.batch) return;             // none of the warp's rows exist
    float sc = p.w_scale;
    if constexpr (SPLIT) sc = j.a0 + ec.q * 32 + ec.lane < p.batch ? p.x_scale[j.a0 + ec.q * 32 + ec.lane] : 0.f;
    const uint64_t scale = pack_f32x2(sc, sc);
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int cb = 128 * ec.h + 64 * half;
      if (cb >= j.n_eff) break;
      const long long col0 = p.lt.row_of(j, j.b0 + cb);
      // (a copy clipped at n_out would still write whole 16-byte pieces)
      const bool by_tma = j.b0 + cb + 64 <= j.rows && col0 + 64 <= p.n_out && (col0 & 7) == 0;
      uint8_t* box = ec.stage + 4096 * (st.boxes % kEpiBoxes);
      if (by_tma) {
        if (ec.lane == 0) {                              // the box has been read by its last store
          if constexpr (kEpiBoxes == 2) bulk_wait_read_but_one();
          else bulk_wait_read_all();
        }
        __syncwarp();
      }
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        const int c0 = cb + 32 * part;
        if (c0 >= j.n_eff) break;                        // warp-uniform
        uint32_t v[32];
        if (have_acc) {
          tmem_ld32(taddr + c0, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0u;
        }
        uint32_t o[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float z0, z1;
          unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), scale), z0, z1);
          o[i] = pack_bf16x2(z0, z1);
        }
        if (by_tma) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            *reinterpret_cast<uint4*>(box + ec.lane * 128 + (((4 * part + i) ^ (ec.lane & 7)) << 4)) =
                make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        } else {
          const int b = j.a0 + ec.q * 32 + ec.lane;
          const long long col = col0 + 32 * part;
          const int valid = b < p.batch ? (int)max(0ll, min(32ll, min((long long)(j.rows - j.b0 - c0), p.n_out - col))) : 0;
          uint16_t* dst = reinterpret_cast<uint16_t*>(p.out) + (size_t)b * p.ld_out + col;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (i < valid) dst[i] = (uint16_t)(o[i >> 1] >> (16 * (i & 1)));
        }
      }
      if (by_tma) {
        fence_proxy_async();
        __syncwarp();
        if (ec.lane == 0) {
          tma_store_2d(ec.map_c, smem_u32(box), (int)col0, j.a0 + ec.q * 32);
          bulk_commit_group();
        }
        ++st.boxes;
      }
    }
  }
};

struct TopkParams {
  int after_prep;          // X was written by the kernel before this one, or by the caller's: every role waits for it
  int own_prep;            // ... this call's preparation of X
  int x_rows;              // rows of a box of X
  int m_rows;              // batch rows per M tile: 128, or 256 on CTA pairs
  int batch;
  int n_mtiles;            // batch tiles of m_rows
  FastDiv div_mtiles;      // of n_mtiles
  LabelTiles lt;           // label tiles of 256
  const CUtensorMap* w_maps;   // one per chunk, in device memory
  long long n_out;         // rows of the handle >= n_out do not count
  int k_steps;
  float w_scale;
  const float* x_scale;    // split embeddings: see FwdParams
  int part_rows;
  const uint8_t* x_wide;
  __nv_bfloat16* out;      // [batch x ld_out], column 0 = this launch's first label row
  long long ld_out;        // multiple of 256
  uint16_t* gmax;          // [batch x ld_gmax] bf16 bits, column 0 = this launch's first 32 labels
  long long ld_gmax;       // multiple of 8
  const float* thr;        // [batch] values that a logit has to exceed, or nullptr while nothing is known
  int* status;
};

// BOX: the first window of a larger batch, whose logits all leave, in boxes of 32 rows x 32 columns by TMA.  (Stored by
// the threads, 32 rows an instruction, they held up the operand converters' shared-memory accesses too; 320 003 x 384 simulated
// FP8, batch 300, 141 -> 129 us.)  A kernel of its own: with both ways in one, and room for the boxes, the windows
// without boxes were up to 7 % slower (1 171 872 x 128 FP8, batch 1 71.3 -> 74.5).  The host's rule has where it pays.
template <bool FP8, Simulated SIM = kSimNone, bool BOX = false>
struct TopkPolicy {
  static constexpr bool SPLIT = SIM == kSimSplit;
  static_assert(SIM == kSimNone || FP8 == SPLIT, "the parts are FP8 operands, the converted weights bf16");
  using Params = TopkParams;
  static constexpr bool kMnMajor = false;
  static constexpr bool kChunkMaps = true;   // Params::w_maps are the maps of one operand or of the epilogue's tile
  static constexpr bool kFp8 = FP8;
  static constexpr uint32_t kFmt = FP8 ? 0u : 1u;
  static constexpr int kElemsPerRow = FP8 ? 128 : 64;
  static constexpr int kEpiWarps = 8;
  static constexpr int kStages = SIM != kSimNone ? 3 : 4;
  static constexpr int kStagesPair = SPLIT ? 4 : kSimConvert == SIM ? 5 : 6;
  static constexpr int kSplit = SPLIT ? 1 : 0, kXRows = 1;
  __device__ static int x_rows(const Params& p) { return p.x_rows; }
  __device__ static int tile_rows(const Params& p) { return p.m_rows; }
  __device__ static int x_tile(const Job& j) { return j.t0; }
  static constexpr bool kConv = SIM == kSimConvert, kEarlyWeights = !kConv;
  static constexpr bool kCTile = false;
  static constexpr int kCBufs = 1;
  static constexpr int kCParts = 1;
  static constexpr bool kBitmap = false;
  static constexpr int kEpiBoxes = SIM != kSimNone ? 1 : 2;      // boxes of 32 rows x 32 columns
  static constexpr int kEpiStage = BOX ? 2048 * kEpiBoxes : 0;
  // Behind the first window the weights and X are written by nothing that may still be running (see FwdPolicy); the
  // epilogue overwrites what the merge before reads.
  static constexpr int kWaitRoles = kRoleEpilogue;
  __device__ static bool wait_all(const Params& p) { return p.after_prep != 0; }
  __device__ static long long wait_limit(const Params&) { return kWaitLimitCycles; }
  __device__ static bool skip_load(const Params&, int, int) { return false; }
  struct EpilogueState {
    uint32_t thr;          // key of the tile's row threshold
    uint32_t boxes;        // boxes stored so far
  };
  __device__ static const CUtensorMap* map_a(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_b(const Params& p, const Job& j, const CUtensorMap*) { return p.w_maps + j.chunk; }
  __device__ static const CUtensorMap* map_c(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static int num_tiles(const Params& p) { return p.n_mtiles * p.lt.count; }
  __device__ static void job(const Params& p, int tile, Job& j) {
    j.t1 = fast_div(tile, p.div_mtiles);  // label tile (adjacent CTAs share it)
    j.t0 = tile - j.t1 * p.n_mtiles;      // batch tile
    j.a0 = j.t0 * p.m_rows;
    j.c_row = j.a0;
    p.lt.locate(j.t1, j, j.b0);
    j.rows = (int)min((long long)j.rows, p.n_out - p.lt.row_of(j, 0));
    j.k_begin = 0;
    j.k_steps = p.k_steps;
    j.n_eff = min(kTileN, max(16, round_up16(j.rows - j.b0)));
  }
  __device__ static void epilogue_begin(const Params&, EpilogueState& st) { st.boxes = 0u; }
  __device__ static void epilogue_prefetch(const Params&, const Job&, EpilogueState&) {}
  __device__ static void epilogue_end(const Params&, SharedTail&, const EpiCtx& ec, EpilogueState&) {
    if constexpr (BOX) {
      if (ec.lane == 0) bulk_wait_all();
      __syncwarp();
    }
  }
  __device__ static void epilogue_pre(const Params& p, const Job& j, SharedTail&, const EpiCtx& ec, EpilogueState& st) {
    if constexpr (BOX) return;
    const int b = j.a0 + ec.q * 32 + ec.lane;
    st.thr = topk_ord16((p.thr != nullptr && b < p.batch) ? __float_as_uint(__ldcg(&p.thr[b])) >> 16 : 0xFF80u);
  }
  __device__ static void epilogue(const Params& p, const Job& j, uint32_t taddr, bool, SharedTail&, const EpiCtx& ec,
                                  EpilogueState& st) {
    if (j.a0 + ec.q * 32 >= p.batch) return;             // none of the warp's rows exist
    const int b = j.a0 + ec.q * 32 + ec.lane;
    const bool active = b < p.batch;
    float sc = p.w_scale;
    if constexpr (SPLIT) sc = active ? p.x_scale[b] : 0.f;
    const uint64_t scale = pack_f32x2(sc, sc);
    constexpr uint32_t kNegInf2 = 0xFF80FF80u;           // bf16x2 (-inf, -inf)
    uint32_t gm[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int c0 = 128 * ec.h + 32 * g;
      const int valid = j.rows - j.b0 - c0;              // warp-uniform
      gm[g] = kNegInf2;
      if (valid <= 0) continue;
      uint32_t v[32];
      tmem_ld32(taddr + c0, v);
      tmem_ld_wait();
      uint32_t o[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float z0, z1;
        unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), scale), z0, z1);
        o[i] = pack_bf16x2(z0, z1);
      }
      if (valid < 32) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (2 * i >= valid) o[i] = kNegInf2;
          else if (2 * i + 1 >= valid) o[i] = (o[i] & 0xFFFFu) | 0xFF800000u;
        }
      }
      // a NaN loses against every number (the maximum of NaNs only becomes -inf): it is never among the best
      uint32_t m = max_bf16x2(o[0], kNegInf2);
#pragma unroll
      for (int i = 1; i < 16; ++i) m = max_bf16x2(m, o[i]);
      m = max_bf16x2(m, __byte_perm(m, m, 0x1032));
      gm[g] = m;
      // equal values of later labels lose; by keys, as the merge reads what it finds above the threshold: as floats +0
      // does not exceed -0, and the merge read logits that had not been written
      if constexpr (BOX) {
        // The first window keeps every logit: a box of 32 columns goes out by TMA.
        uint8_t* box = ec.stage + 2048 * (st.boxes % kEpiBoxes);
        if (ec.lane == 0) {                                // the box has been read by its last store
          if constexpr (kEpiBoxes == 2) bulk_wait_read_but_one();
          else bulk_wait_read_all();
        }
        __syncwarp();
        // 64-byte rows, 16-byte pieces XOR half the row (the 64-byte swizzle of the copy)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          *reinterpret_cast<uint4*>(box + ec.lane * 64 + ((i ^ ((ec.lane >> 1) & 3)) << 4)) =
              make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        fence_proxy_async();
        __syncwarp();
        if (ec.lane == 0) {
          tma_store_2d(ec.map_c, smem_u32(box), j.t1 * kTileN + c0, j.a0 + ec.q * 32);
          bulk_commit_group();
        }
        ++st.boxes;
      } else if (active && topk_ord16(m & 0xFFFFu) > st.thr) {
        __nv_bfloat16* dst = p.out + (size_t)b * p.ld_out + j.t1 * kTileN + c0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          U32x8 o8;
#pragma unroll
          for (int k = 0; k < 8; ++k) o8.v[k] = o[8 * i + k];
          st_global_256(dst + 16 * i, o8);
        }
      }
    }
    if (active)
      *reinterpret_cast<uint2*>(p.gmax + (size_t)b * p.ld_gmax + j.t1 * (kTileN / 32) + 4 * ec.h) =
          make_uint2(__byte_perm(gm[0], gm[1], 0x5410), __byte_perm(gm[2], gm[3], 0x5410));
  }
};

// -------------------------------------------------------------------------------------------------
// Plain D = A B^T, fp32 out (engine self-test; also the logits kernel's skeleton)
// -------------------------------------------------------------------------------------------------
struct PlainParams {
  int m_rows;              // rows per M tile (128)
  int M, N;
  int n_mtiles, n_ntiles;
  int k_steps;
  float* D;                // [M x N]
  int checksum_only;       // 1: do not store D (times the main loop without the output traffic)
  long long test_wait_limit;   // > 0: every wait of the kernel gives up after this many cycles
  int test_skip_tile;      // the producer leaves out the second k-step of this tile (-1: none)
  int* status;
};

template <bool FP8, bool MN>
struct PlainPolicy {
  using Params = PlainParams;
  static constexpr bool kMnMajor = MN;
  static constexpr bool kChunkMaps = false;
  static constexpr bool kFp8 = FP8;
  static constexpr uint32_t kFmt = FP8 ? 0u : 1u;
  static constexpr int kElemsPerRow = FP8 ? 128 : 64;
  static constexpr int kEpiWarps = 8;
  static constexpr int kStages = 4;
  static constexpr int kStagesPair = 6;
  static constexpr int kSplit = 0, kXRows = 0;
  __device__ static int x_rows(const Params&) { return 0; }
  static constexpr bool kConv = false, kEarlyWeights = false;
  static constexpr bool kCTile = false;
  static constexpr int kCBufs = 1;
  static constexpr int kCParts = 1;
  static constexpr bool kBitmap = false;
  static constexpr int kEpiStage = 0;
  static constexpr int kWaitRoles = kRoleAll;
  // failure-injection of the self-test: a shortened wait limit and one operand load left out
  __device__ static bool wait_all(const Params&) { return true; }
  __device__ static long long wait_limit(const Params& p) { return p.test_wait_limit > 0 ? p.test_wait_limit : kWaitLimitCycles; }
  __device__ static bool skip_load(const Params& p, int tile, int k) { return tile == p.test_skip_tile && k == 1; }
  using EpilogueState = NoState;
  __device__ static const CUtensorMap* map_a(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_b(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static const CUtensorMap* map_c(const Params&, const Job&, const CUtensorMap* m) { return m; }
  __device__ static int num_tiles(const Params& p) { return p.n_mtiles * p.n_ntiles; }
  __device__ static void job(const Params& p, int tile, Job& j) {
    j.t0 = tile / p.n_ntiles;
    j.t1 = tile - j.t0 * p.n_ntiles;
    j.a0 = j.t0 * p.m_rows;
    j.b0 = j.t1 * kTileN;
    j.c_row = j.a0;
    j.chunk = 0;
    j.rows = p.M;
    j.k_begin = 0;
    j.k_steps = p.k_steps;
    j.n_eff = min(kTileN, round_up16(p.N - j.b0));
  }
  __device__ static void epilogue_begin(const Params&, EpilogueState&) {}
  __device__ static void epilogue_pre(const Params&, const Job&, SharedTail&, const EpiCtx&, EpilogueState&) {}
  __device__ static void epilogue_prefetch(const Params&, const Job&, EpilogueState&) {}
  __device__ static void epilogue_end(const Params&, SharedTail&, const EpiCtx&, EpilogueState&) {}
  __device__ static void epilogue(const Params& p, const Job& j, uint32_t taddr, bool have_acc,
                                  SharedTail&, const EpiCtx& ec, EpilogueState&) {
    const int m = j.a0 + ec.q * 32 + ec.lane;
    for (int c0 = 32 * ec.h; c0 < j.n_eff; c0 += 32 * ec.nsplit) {
      uint32_t v[32];
      if (have_acc) {
        tmem_ld32(taddr + c0, v);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0u;
      }
      if (m >= p.M) continue;
      if (p.checksum_only) {          // main-loop timing: fold the tile into one word per thread
        uint32_t x = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) x ^= v[i];
        if (x == 0x12345678u) p.D[0] = 1.f;
        continue;
      }
      float* drow = p.D + (size_t)m * p.N + j.b0 + c0;
      if ((p.N & 3) == 0 && j.b0 + c0 + 32 <= p.N) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          reinterpret_cast<float4*>(drow)[i] = make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                                           __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (j.b0 + c0 + i < p.N) drow[i] = __uint_as_float(v[i]);
      }
    }
  }
};

}  // namespace xmc
