// Bandwidth-bound helper kernels around the GEMMs: embedding preparation, bucketing of the sparse
// positives by label tile, the merge of the top-k windows, and the fixed-order final reductions.
#pragma once
#include "numerics.cuh"
#include "ptx.cuh"

namespace xmc {

// All helper kernels are launched with programmatic stream serialization (ptx.cuh).  Three rules make it safe that some
// roles of the big kernels read without waiting (the weights, written a step ago, and X as prepared here): every
// kernel waits for its predecessor before it ends; a helper lets its successor start only after its own wait,
// so whatever runs behind it finds all earlier calls complete; and the kernels that prepare X let it start only when
// X is written and visible, because the kernel after next may already run by then.

// X [batch x d] (bf16 or e4m3) -> x8 [rows8 x d] e4m3, x16 [rows16 x d] bf16, xt [d x bpad] bf16.
// Rows/columns in [batch, bpad) are written as zero.  32x32 tiles through shared memory so that
// both the row-major and the transposed stores are coalesced.
struct PrepX {
  const void* x;
  int batch, bpad, d;
  uint8_t* x8;
  __nv_bfloat16* x16;
  __nv_bfloat16* xt;
  uint8_t* xt8;
  // Split embeddings ("simulated FP8": bf16 embeddings by e4m3 weights, on the FP8 tensor cores), or nullptr: four arrays
  // part_bytes apart, parts 0 and 2 in e4m3, 1 and 3 in e5m2.  (With parts 0 and 2 of a row side by side, and 1 and 3, the rows twice as far apart, top
  // 10 of 320 003 x 384 for 300 rows took 130 instead of 127 us.)  A row is multiplied by the power of two that brings its largest
  // number into [128, 256); part 0 takes that rounded to e4m3, four significant bits, part 1 the rest, which is e5m2 with its three
  // bits: bf16 has eight, and the sign of the rest is one.  Exact down to 2^-13 of the row's largest, where part 0 has its four
  // bits; what is smaller comes within 2^-21 of that largest.  Where all that is lacking is more than 2^-24 of the row's
  // magnitudes, summed up -- as much as rounding a sum of fp32 once -- the row is wide: its largest comes into [2^14, 2^15), part 0
  // takes what is below 256, and parts 1, 3 and 2, in that order, what is left: exact down to 2^-23 of the largest (where a number
  // has all its bits in multiples of 2^-16, e5m2's smallest), within 2^-31 of it below.  Parts 2 and 3 are multiplied for tiles with a
  // wide row only, and hold zeros for other rows, always.  Infinities sit in part 1, a NaN in part 0.
  // x_scale: what the kernels multiply the accumulators of the row by, w_scale over that power of two.
  uint8_t* parts;
  size_t part_bytes;
  uint8_t* x_wide;         // by row; kept from call to call, as are parts 2 and 3, which a row that is wide no longer clears
  float* x_scale;
  float w_scale;
  int row_blocks;          // blocks that split embeddings, a row a warp; those with a 32 x 32 tile of X follow
};
// A warp's row b: read once, in one piece up to 1024 features.  Eight rows a block: with a row for each of 32 warps a call that
// waits for a few rows took 3 us longer.
constexpr int kSplitRows = 8;
__device__ __forceinline__ void split_row(const PrepX& p, int b) {
  const int lane = threadIdx.x & 31, n8 = p.d / 8;
  const uint16_t* row = reinterpret_cast<const uint16_t*>(p.x) + (size_t)b * p.d;
  const bool aligned = (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0;       // rows are multiples of 128 bytes
  const int there = b < p.batch ? n8 : 0;
  auto eight = [&](int i) {
    const uint16_t* e = row + 8 * i;
    return make_uint4(e[0] | ((uint32_t)e[1] << 16), e[2] | ((uint32_t)e[3] << 16), e[4] | ((uint32_t)e[5] << 16), e[6] | ((uint32_t)e[7] << 16));
  };
  auto fetch = [&](int i0, uint4 (&r)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = make_uint4(0u, 0u, 0u, 0u);
    if (aligned) {                                           // all of them under way at a time
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + lane + 32 * u < there) r[u] = reinterpret_cast<const uint4*>(row)[i0 + lane + 32 * u];
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + lane + 32 * u < there) r[u] = eight(i0 + lane + 32 * u);
    }
  };
  const bool was_wide = p.x_wide[b] != 0;
  uint32_t m = 0u;                                           // the largest magnitude among the finite ones
  auto take = [&](uint32_t bits) { bits &= 0x7FFFu; m = bits < 0x7F80u ? max(m, bits) : m; };
  uint4 r[4];
  for (int i0 = 0; i0 < n8; i0 += 128) {
    fetch(i0, r);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      take(r[u].x); take(r[u].x >> 16); take(r[u].y); take(r[u].y >> 16);
      take(r[u].z); take(r[u].z >> 16); take(r[u].w); take(r[u].w >> 16);
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  // 2^(e - 127) <= m: k = 7 - (e - 127), as far as a normal number's reciprocal goes
  const int k = m == 0u ? 0 : min(134 - max(1, (int)(m >> 7)), 126);
  const float scale = __int_as_float((127 + k) << 23);
  uint8_t* const part = p.parts + (size_t)b * p.d;
  float all = 0.f, lacking = 0.f;
  for (int i0 = 0; i0 < n8; i0 += 128) {
    if (n8 > 128) fetch(i0, r);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + lane + 32 * u;
      if (i >= n8) continue;
      const uint32_t w[4] = {r[u].x, r[u].y, r[u].z, r[u].w};
      uint32_t hi[2] = {0u, 0u}, lo[2] = {0u, 0u};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float v0 = __uint_as_float(w[e] << 16), v1 = __uint_as_float(w[e] & 0xFFFF0000u);
        const float x0 = v0 * scale, x1 = v1 * scale;
        uint32_t h = float2_to_e4m3x2(x0, x1);
        const float2 f = e4m3x2_to_float2((uint16_t)h);
        uint32_t l = (uint32_t)__nv_cvt_float2_to_fp8x2(make_float2(x0 - f.x, x1 - f.y), __NV_SATFINITE, __NV_E5M2);
        float got[4];
        e5m2x4_to_float4(l, got);
        if (fabsf(v0) < INFINITY) {
          all += fabsf(x0);
          lacking += fabsf(x0 - f.x - got[0]);
        } else {
          h = (h & 0xFF00u) | (v0 != v0 ? 0x7Fu : 0u);
          l = (l & 0xFF00u) | (v0 != v0 ? 0u : v0 > 0.f ? 0x7Cu : 0xFCu);
        }
        if (fabsf(v1) < INFINITY) {
          all += fabsf(x1);
          lacking += fabsf(x1 - f.y - got[1]);
        } else {
          h = (h & 0xFFu) | (v1 != v1 ? 0x7F00u : 0u);
          l = (l & 0xFFu) | (v1 != v1 ? 0u : v1 > 0.f ? 0x7C00u : 0xFC00u);
        }
        hi[e >> 1] |= h << (16 * (e & 1));
        lo[e >> 1] |= l << (16 * (e & 1));
      }
      reinterpret_cast<uint2*>(part)[i] = make_uint2(hi[0], hi[1]);
      reinterpret_cast<uint2*>(part + p.part_bytes)[i] = make_uint2(lo[0], lo[1]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    all += __shfl_xor_sync(0xffffffffu, all, o);
    lacking += __shfl_xor_sync(0xffffffffu, lacking, o);
  }
  const bool wide = lacking * 16777216.f > all;
  const int kw = wide ? min(k + 7, 126) : k;
  if (lane == 0) {
    p.x_scale[b] = p.w_scale * __int_as_float((127 - kw) << 23);
    p.x_wide[b] = wide ? 1 : 0;
  }
  if (!wide && !was_wide) return;
  const float wide_scale = __int_as_float((127 + kw) << 23);
#pragma unroll 1
  for (int i = lane; i < n8; i += 32) {
    const uint4 r8 = i >= there ? make_uint4(0u, 0u, 0u, 0u) : aligned ? reinterpret_cast<const uint4*>(row)[i] : eight(i);
    const uint32_t w[4] = {r8.x, r8.y, r8.z, r8.w};
    uint32_t got[4][2] = {{0u, 0u}, {0u, 0u}, {0u, 0u}, {0u, 0u}};
    if (wide) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float v = __uint_as_float((e & 1) ? w[e >> 1] & 0xFFFF0000u : w[e >> 1] << 16);
        float rest = fabsf(v) < INFINITY ? v * wide_scale : 0.f;
        auto take = [&](int j, uint32_t bits, float value) {
          got[j][e >> 2] |= bits << (8 * (e & 3));
          rest -= value;
        };
        auto e4m3 = [&](int j) {
          const uint32_t l = float2_to_e4m3x2(rest, 0.f) & 0xFFu;
          take(j, l, e4m3x2_to_float2((uint16_t)l).x);
        };
        auto e5m2 = [&](int j) {
          const uint32_t l = (uint32_t)__nv_cvt_float_to_fp8(rest, __NV_SATFINITE, __NV_E5M2);
          float f[4];
          e5m2x4_to_float4(l, f);
          take(j, l, f[0]);
        };
        if (fabsf(rest) < 256.f) e4m3(0);
        e5m2(1);
        e5m2(3);
        e4m3(2);
        if (v != v) take(0, 0x7Fu, 0.f);
        else if (!(fabsf(v) < INFINITY)) take(1, v > 0.f ? 0x7Cu : 0xFCu, 0.f);
      }
      reinterpret_cast<uint2*>(part)[i] = make_uint2(got[0][0], got[0][1]);
      reinterpret_cast<uint2*>(part + p.part_bytes)[i] = make_uint2(got[1][0], got[1][1]);
    }
    reinterpret_cast<uint2*>(part + 2 * p.part_bytes)[i] = make_uint2(got[2][0], got[2][1]);
    reinterpret_cast<uint2*>(part + 3 * p.part_bytes)[i] = make_uint2(got[3][0], got[3][1]);
  }
}
// An element a thread: with 256 threads, four each, a call that waits for its embeddings takes longer (top-k of 200 000 x 768 at
// batch 64 46.0 and 44.4 us, logits of 131 072 x 768 at 64 26.8 and 25.6).
constexpr int kPrepThreads = 1024;
template <bool IN_E4M3, int THREADS>
__device__ __forceinline__ void prep_x_tile(const PrepX& p, int c0, int b0) {
  __shared__ float tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int i = ty; i < 32; i += THREADS / 32) {
    const int b = b0 + i, c = c0 + tx;
    float v = 0.f;
    if (b < p.batch && c < p.d) {
      if (IN_E4M3) {
        const uint8_t raw = reinterpret_cast<const uint8_t*>(p.x)[(size_t)b * p.d + c];
        v = e4m3x2_to_float2((uint16_t)raw).x;
      } else {
        v = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.x)[(size_t)b * p.d + c]);
      }
    }
    tile[i][tx] = v;
    if (b < p.bpad && c < p.d) {
      if (IN_E4M3 && p.parts != nullptr) {                   // e4m3 embeddings, to be split: as they are, and no rest
        p.parts[p.part_bytes + (size_t)b * p.d + c] = 0;
        if (c == 0) p.x_scale[b] = p.w_scale;
      }
      if (p.x8 != nullptr) p.x8[(size_t)b * p.d + c] = (uint8_t)(float2_to_e4m3x2(v, 0.f) & 0xFFu);
      if (p.x16 != nullptr) p.x16[(size_t)b * p.d + c] = __float2bfloat16_rn(v);
    }
  }
  __syncthreads();
  if (p.xt != nullptr || p.xt8 != nullptr) {
    for (int i = ty; i < 32; i += THREADS / 32) {
      const int c = c0 + i, b = b0 + tx;
      if (c < p.d && b < p.bpad) {
        if (p.xt != nullptr) p.xt[(size_t)c * p.bpad + b] = __float2bfloat16_rn(tile[tx][i]);
        if (p.xt8 != nullptr) p.xt8[(size_t)c * p.bpad + b] = (uint8_t)(float2_to_e4m3x2(tile[tx][i], 0.f) & 0xFFu);
      }
    }
  }
}
// SPLIT: embeddings to be split.  Kernels of their own: with 53 registers instead of 32 no two blocks of 1024 threads share an SM, and the
// headline step's preparation (670 091 x 768, batch 512) takes 15.4 us instead of 13.6.
template <bool IN_E4M3, int THREADS, bool SPLIT>
__device__ __forceinline__ void prep_x_block(const PrepX& p, int t) {
  const int row_blocks = SPLIT ? p.row_blocks : 0;
  if (t < row_blocks) {
    const int b = t * kSplitRows + (int)(threadIdx.x >> 5);
    if ((int)(threadIdx.x >> 5) < kSplitRows && b < p.bpad) split_row(p, b);
  } else {
    const int n_ct = (p.d + 31) / 32;
    t -= row_blocks;
    prep_x_tile<IN_E4M3, THREADS>(p, (t % n_ct) * 32, (t / n_ct) * 32);
  }
}
template <bool IN_E4M3, bool SPLIT>
__global__ void __launch_bounds__(kPrepThreads)
prep_x_kernel(const PrepX p, int early) {
  pdl_wait();
  if (early) pdl_launch_dependents();
  prep_x_block<IN_E4M3, kPrepThreads, SPLIT>(p, (int)blockIdx.x);
  __threadfence();
  pdl_launch_dependents();
}

// ---------------------------------------------------------------------------------------------
// Positives (row, global label id) -> buckets of 128 label rows, chunk after chunk.
// ---------------------------------------------------------------------------------------------
struct BucketGeom {
  long long label_offset;   // global id of the handle's row 0
  long long total_rows;
  int rows_per_chunk;       // rows of every bound weight chunk but the last
  int per_chunk;            // buckets of a chunk
  int n_buckets;
};

__device__ __forceinline__ bool bucket_of(const BucketGeom& g, int row, int col, int batch, int* status,
                                          int& bucket, int& lrow) {
  if (row < 0 || row >= batch || col < 0) {
    report(status, DEV_BAD_LABEL, row);
    return false;
  }
  const long long r = (long long)col - g.label_offset;
  if (r < 0 || r >= g.total_rows) return false;          // another shard's label
  const unsigned int wc = (unsigned int)r / (unsigned int)g.rows_per_chunk;    // a handle has fewer than 2^31 rows
  const unsigned int in = (unsigned int)r - wc * (unsigned int)g.rows_per_chunk;
  bucket = (int)wc * g.per_chunk + (int)(in >> 7);
  lrow = (int)(in & 127u);
  return true;
}

// One more in `count` of a bucket, in global memory, for every lane with one (bucket >= 0), and the count before it.  Lanes of
// the same bucket go together: popular labels share one, and 32 lanes at the same word are 32 turns.  Preparation of a step
// with 49 132 pairs of 100 000 labels (Zipf 1.1) 76 -> 47 us, with 24 479 51 -> 34.
__device__ __forceinline__ int bucket_add(int* count, int bucket, int lane) {
  const unsigned int same = __match_any_sync(0xffffffffu, bucket);
  int before = 0;
  if (bucket >= 0 && lane == __ffs(same) - 1) before = atomicAdd(&count[bucket], __popc(same));
  return __shfl_sync(0xffffffffu, before, __ffs(same) - 1) + __popc(same & ((1u << lane) - 1u));
}

__global__ void bucket_count_kernel(const int32_t* __restrict__ labels, long long nnz, int batch,
                                    BucketGeom g, int* __restrict__ count, int* status) {
  pdl_wait();
  pdl_launch_dependents();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int bucket = -1, lrow;
  if (i >= nnz || !bucket_of(g, labels[2 * i], labels[2 * i + 1], batch, status, bucket, lrow)) bucket = -1;
  bucket_add(count, bucket, threadIdx.x & 31);
}

// exclusive scan of count[0..n) into off[0..n], single block
__global__ void bucket_scan_kernel(const int* __restrict__ count, int n, int* __restrict__ off) {
  pdl_wait();
  pdl_launch_dependents();
  __shared__ int warp_sum[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = 0; base < n; base += blockDim.x) {
    const int i = base + threadIdx.x;
    const int v = i < n ? count[i] : 0;
    int s = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    if (lane == 31) warp_sum[warp] = s;
    __syncthreads();
    if (warp == 0) {
      int w = lane < (int)(blockDim.x >> 5) ? warp_sum[lane] : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
      }
      warp_sum[lane] = w;
    }
    __syncthreads();
    const int before = carry + (warp > 0 ? warp_sum[warp - 1] : 0) + s - v;
    if (i < n) off[i] = before;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) off[n] = carry;
}

__global__ void bucket_fill_kernel(const int32_t* __restrict__ labels, long long nnz, int batch,
                                   BucketGeom g, const int* __restrict__ off, int* __restrict__ cursor,
                                   uint32_t* __restrict__ entries) {
  pdl_wait();
  pdl_launch_dependents();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int bucket = -1, lrow = 0;
  const int row = i < nnz ? labels[2 * i] : 0;
  if (i >= nnz || !bucket_of(g, row, labels[2 * i + 1], batch, nullptr, bucket, lrow)) bucket = -1;
  const int pos = bucket_add(cursor, bucket, threadIdx.x & 31);
  if (bucket >= 0) entries[off[bucket] + pos] = (uint32_t)row | ((uint32_t)lrow << 16);
}

// Count, scan and fill by ONE block.
// The counts of all buckets live in shared memory (s_off, n + 1 words): counting and filling are shared-memory
// atomics (with the counts in global memory three times slower), a pair each.  (Lanes of the same bucket going together, as
// above, cost more than the turns they save here: step of 4 001 x 256 at batch 128 with 2 200 pairs 23.0 us and 21.2.)
template <int THREADS, int KEEP>
__device__ __forceinline__ void bucket_block(const int32_t* __restrict__ labels, int nnz, int batch, const BucketGeom& g,
                                             int* off, uint32_t* __restrict__ entries, int* status, int* s_off) {
  __shared__ int warp_sum[THREADS / 32];
  const int n = g.n_buckets;
  for (int i = threadIdx.x; i <= n; i += THREADS) s_off[i] = 0;
  __syncthreads();
  // Several pairs in flight per thread: the loads' latency is what the two passes consist of.  Where a thread has no more
  // than KEEP pairs, the first pass keeps their places for the second.
  constexpr int kAhead = 8;
  const bool kept = nnz <= KEEP * THREADS;
  int at[KEEP > 0 ? KEEP : 1];                               // bucket, -1: none
  uint32_t ent[KEEP > 0 ? KEEP : 1];
  for (int i0 = threadIdx.x; i0 < nnz; i0 += kAhead * THREADS) {
    int2 pair[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (i0 + u * THREADS < nnz) pair[u] = reinterpret_cast<const int2*>(labels)[i0 + u * THREADS];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      int bucket, lrow;
      const bool ok = i0 + u * THREADS < nnz && bucket_of(g, pair[u].x, pair[u].y, batch, status, bucket, lrow);
      if (ok) atomicAdd(&s_off[bucket], 1);
      if (u < KEEP) {
        at[u] = ok ? bucket : -1;
        ent[u] = (uint32_t)pair[u].x | ((uint32_t)lrow << 16);
      }
    }
  }
  __syncthreads();
  // exclusive scan: every thread sums a contiguous run of buckets, one block-wide scan of the run totals, then
  // each thread turns the counts of its run into offsets
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (n + THREADS - 1) / THREADS;
  const int beg = min(n, (int)threadIdx.x * per), end = min(n, beg + per);
  int run = 0;
  for (int i = beg; i < end; ++i) run += s_off[i];
  int s = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += t;
  }
  if (lane == 31) warp_sum[warp] = s;
  __syncthreads();
  int before = s - run;
  for (int w = 0; w < warp; ++w) before += warp_sum[w];
  for (int i = beg; i < end; ++i) {
    const int c = s_off[i];
    s_off[i] = before;
    before += c;
  }
  if (threadIdx.x == THREADS - 1) s_off[n] = before;        // the last thread's run ends at n (or is empty)
  __syncthreads();
  for (int i = threadIdx.x; i <= n; i += THREADS) off[i] = s_off[i];
  __syncthreads();
  if (KEEP > 0 && kept) {
    if ((int)threadIdx.x < nnz) {
#pragma unroll
      for (int u = 0; u < KEEP; ++u)
        if (at[u] >= 0) entries[atomicAdd(&s_off[at[u]], 1)] = ent[u];
    }
    return;
  }
  for (int i0 = threadIdx.x; i0 < nnz; i0 += kAhead * THREADS) {
    int2 pair[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (i0 + u * THREADS < nnz) pair[u] = reinterpret_cast<const int2*>(labels)[i0 + u * THREADS];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      int bucket, lrow;
      if (i0 + u * THREADS >= nnz) break;
      if (bucket_of(g, pair[u].x, pair[u].y, batch, nullptr, bucket, lrow))
        entries[atomicAdd(&s_off[bucket], 1)] = (uint32_t)pair[u].x | ((uint32_t)lrow << 16);
    }
  }
}

// The preparation of a whole step in one launch: block 0 sorts the positives into buckets, the others take a 32 x 32
// tile of X each.  early: every role of the kernel behind waits for this one, which may then start at once.
//
// KEEP > 0: pairs that a thread keeps between the two passes of the sort, for 16 registers more (steps of 4 001 x 768, batch 64, with
// 1 900 pairs 24.1 -> 22.5 us, with 500 22.0 -> 21.4).  Beyond batch 128 the blocks with X are what is waited for, and
// two of them share an SM without (31 003 x 768, batch 256 59.4 and 59.9).
template <int THREADS, int KEEP, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
prep_step_kernel(const PrepX p, const int32_t* __restrict__ labels, int nnz, const BucketGeom g, int* off,
                 uint32_t* __restrict__ entries, int* status, int early) {
  extern __shared__ int prep_smem[];
  pdl_wait();
  if (early) pdl_launch_dependents();
  if (blockIdx.x == 0) {
    bucket_block<THREADS, KEEP>(labels, nnz, p.batch, g, off, entries, status, prep_smem);
  } else {
    prep_x_block<false, THREADS, SPLIT>(p, (int)blockIdx.x - 1);
  }
  __threadfence();
  pdl_launch_dependents();
}

// Scale bookkeeping: one streaming pass over e4m3 weights (n16 groups of 16 bytes).
// counts[0] zeros, [1] sub-normal magnitudes (0 < |w| < 2^-6), [2] at +-448, [3] NaN; amax_bits = largest
// magnitude byte seen (e4m3 magnitudes order like their bytes).
__global__ void weight_stats_kernel(const uint4* __restrict__ w, long long n16, unsigned long long* counts,
                                    unsigned int* amax_bits) {
  unsigned int zeros = 0, sub = 0, sat = 0, nan = 0, amax = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) {
    const uint4 raw = w[i];
    const uint32_t ws[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const unsigned int m = (ws[k] >> (8 * b)) & 0x7Fu;
        zeros += m == 0u;
        sub += (m != 0u) & (m < 0x08u);
        sat += m == 0x7Eu;
        nan += m == 0x7Fu;
        amax = max(amax, m == 0x7Fu ? 0u : m);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    zeros += __shfl_xor_sync(0xffffffffu, zeros, o);
    sub += __shfl_xor_sync(0xffffffffu, sub, o);
    sat += __shfl_xor_sync(0xffffffffu, sat, o);
    nan += __shfl_xor_sync(0xffffffffu, nan, o);
    amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  }
  if ((threadIdx.x & 31) == 0) {
    if (zeros) atomicAdd(&counts[0], (unsigned long long)zeros);
    if (sub) atomicAdd(&counts[1], (unsigned long long)sub);
    if (sat) atomicAdd(&counts[2], (unsigned long long)sat);
    if (nan) atomicAdd(&counts[3], (unsigned long long)nan);
    atomicMax(amax_bits, amax);
  }
}

// stored <- round(stored * factor) for a power-of-two factor (the per-tensor scale moves the other way).
// Growing is exact up to saturation at +-448; shrinking rounds what falls below the grid: to nearest, or
// stochastically with the step's Philox stream (counter = global element index / 8, as in the update).
__global__ void rescale_e4m3_kernel(uint2* __restrict__ w, long long n8, float factor, int stochastic,
                                    unsigned long long seed, unsigned long long step, unsigned long long elem0) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += stride) {
    const uint2 raw = w[i];
    const uint32_t rw[2] = {raw.x, raw.y};
    uint4 r = make_uint4(0u, 0u, 0u, 0u);
    if (stochastic) {
      const unsigned long long q = (elem0 >> 3) + (unsigned long long)i;
      r = philox4x32_sr(make_uint4((uint32_t)q, (uint32_t)(q >> 32), (uint32_t)step, (uint32_t)(step >> 32)),
                        make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    }
    const uint32_t rr[4] = {r.x, r.y, r.z, r.w};
    uint32_t ow[2] = {0u, 0u};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      float v = e4m3x2_to_float2((uint16_t)(rw[e >> 2] >> (8 * (e & 3)))).x * factor;
      if (stochastic) v = sr_e4m3(v, (e & 1) ? (rr[e >> 1] >> 16) : (rr[e >> 1] & 0xFFFFu));
      ow[e >> 2] |= ((uint32_t)float2_to_e4m3x2(v, 0.f) & 0xFFu) << (8 * (e & 3));
    }
    w[i] = make_uint2(ow[0], ow[1]);
  }
}

// out[i] = bf16(sigmoid(in[i])) exactly as the forward epilogue computes it (test hook)
__global__ void sigmoid_probe_kernel(const __nv_bfloat16* __restrict__ in, __nv_bfloat16* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16_rn(fast_sigmoid(__bfloat162float(in[i])));
}

// grad_X[b][c] = scale * sum_s partial[s][b][c] in a fixed order.  A block takes 32 runs of four columns; its eight
// warps take the slots w, w + 8, ... with several loads in flight, and the eight sums meet in shared memory.  Bound by
// the read of the partial sums from L2.  (One thread per element walking all slots one after the other was
// bound by the latency of 74 dependent turns: 11 us at batch 32 x 768, now 4.)
//
// Where the loss is asked for the last block sums it up, beside the others: a fixed order, thread t adds partials t, t + 256,
// ..., eight loads at a time, and the sums meet in a tree; bound by the latency of its n / 2048 trips.  (A launch of its own
// behind this one was 3 us of a small step: 31 003 x 512, batch 100 with loss 72.3 -> 69.5.)
constexpr int kReduceThreads = 256;
struct LossSum {
  const double* partial;
  int n;                   // partials; 0: no loss is asked for
  double* out;
};
__device__ __forceinline__ void reduce_loss(const LossSum& l) {
  __shared__ double warp_sum[kReduceThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s = 0.0;
#pragma unroll 8
  for (int i = threadIdx.x; i < l.n; i += kReduceThreads) s += __ldcg(&l.partial[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) warp_sum[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    s = warp_sum[0];
    for (int w = 1; w < kReduceThreads / 32; ++w) s += warp_sum[w];
    *l.out = s;
  }
}
__global__ void __launch_bounds__(kReduceThreads)
reduce_gradx_kernel(const float* __restrict__ partial, int n_splits, int batch, int slot_rows, int d, float scale,
                    float* __restrict__ out32, __nv_bfloat16* __restrict__ out16, const LossSum loss) {
  __shared__ float4 part[kReduceThreads / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long n4 = (long long)batch * d / 4;             // d is a multiple of 64
  const long long slot4 = (long long)slot_rows * d / 4;
  pdl_wait();
  pdl_launch_dependents();
  const int blocks = (int)gridDim.x - (loss.n > 0 ? 1 : 0);
  if ((int)blockIdx.x == blocks) {
    reduce_loss(loss);
    return;
  }
  for (long long i0 = (long long)blockIdx.x * 32; i0 < n4; i0 += (long long)blocks * 32) {
    const long long i = i0 + lane;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n4) {
      const float4* src = reinterpret_cast<const float4*>(partial) + i;
#pragma unroll 4
      for (int k = warp; k < n_splits; k += kReduceThreads / 32) {
        const float4 v = __ldcg(src + k * slot4);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && i < n4) {
#pragma unroll
      for (int w = 1; w < kReduceThreads / 32; ++w) {
        const float4 v = part[w][lane];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
      s.x *= scale; s.y *= scale; s.z *= scale; s.w *= scale;
      if (out32 != nullptr) reinterpret_cast<float4*>(out32)[i] = s;
      if (out16 != nullptr) {
        __nv_bfloat16* o = out16 + 4 * i;
        if ((reinterpret_cast<uintptr_t>(out16) & 7u) == 0) {
          *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16x2(s.x, s.y), pack_bf16x2(s.z, s.w));
        } else {                                             // the caller's tensor may start at any element
          o[0] = __float2bfloat16_rn(s.x); o[1] = __float2bfloat16_rn(s.y);
          o[2] = __float2bfloat16_rn(s.z); o[3] = __float2bfloat16_rn(s.w);
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------------
// Top-k of one batch row over one more window of labels, one block per row.  In: the largest logit of every
// 32 labels of the window (gmax) and, where that maximum exceeds the row's threshold, the 32 logits
// themselves (z); the k best of the windows before (run).  Out: the k best so far and the new threshold, or,
// after the last window, the result.
//
// Candidates are the logits of the window at or above a bound: the next value after the old threshold
// or, where that lets through many groups (the first window), the k-th largest of the maxima -- k different
// labels reach it, so it bounds the k-th best value from below, and only about k groups reach it.
// A candidate becomes a 64-bit key (ordered value, ~label): larger key = larger value and, among equal values,
// the lower label; labels are unique, hence keys are.  Logits are bf16, so 16 bits decide about values.  Up to
// kTopkList keys are ranked by counting the larger ones (each key compared with all others: the rank is
// also the place in the output); of more, the value or the key of the k-th largest is first found two bits
// at a time.  Keys that do not fit into shared memory (thousands of equal logits) are visited in global memory instead.
//
// Latency-bound: a few dependent trips to L2 and a handful of block-wide steps, three to five microseconds a window.  What
// is read from global memory is therefore asked for at once, groups are listed while their maxima come in, and the
// bound of a first window (eight rounds over the block, which were 13 of its 29 thousand cycles) looks at the
// threads' own maxima.  Selecting the best of a window without ranking them costs more rounds than it saves
// (eight rounds against 130 comparisons a thread: top 100 of 670 208 x 512 287 -> 311 us).
// ---------------------------------------------------------------------------------------------
constexpr int kTopkThreads = 256;
constexpr int kTopkMaxK = 128;
constexpr int kTopkCand = 4096;          // candidates held in shared memory
constexpr int kTopkList = 512;           // candidates ranked directly
constexpr int kTopkHits = 1024;          // groups listed
constexpr int kTopkMaxGroups = 16384;    // groups of 32 labels per window

__device__ __forceinline__ unsigned long long topk_key64(float v, int id) {
  const unsigned int bits = __float_as_uint(v);
  const unsigned int ord = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
  return ((unsigned long long)ord << 32) | (unsigned long long)(0xFFFFFFFFu - (unsigned int)id);
}
__device__ __forceinline__ float topk_value(unsigned long long key) {
  const unsigned int ord = (unsigned int)(key >> 32);
  return __uint_as_float((ord & 0x80000000u) ? (ord & 0x7FFFFFFFu) : ~ord);
}

struct TopkMerge {
  const uint16_t* gmax;     // [batch x ld_gmax]
  long long ld_gmax;
  const __nv_bfloat16* z;   // [batch x ld_z]
  long long ld_z;
  int n_groups;             // groups of the window
  int first_group;          // the window's first group in the list of all chunks' groups ...
  int chunk_groups;         // ... of which every chunk but the last has this many, for
  int chunk_rows;           // this many labels
  long long label0;         // global id of the handle's first label
  int k, first, last;       // first / last window of the call
  unsigned long long* run;  // [batch x kTopkMaxK]
  int* run_cnt;             // [batch]
  float* thr;               // [batch]
  float* out_val;           // [batch x k]
  int* out_idx;
};
__host__ __device__ constexpr int topk_smem_bytes(int n_groups) {
  return kTopkCand * 8 + kTopkList * 8 + kTopkHits * 4 + (n_groups + 7) / 8 * 16;
}

__global__ void __launch_bounds__(kTopkThreads)
topk_merge_kernel(const TopkMerge p) {
  extern __shared__ __align__(16) unsigned char topk_smem[];
  unsigned long long* cand = reinterpret_cast<unsigned long long*>(topk_smem);
  unsigned long long* list = cand + kTopkCand;
  int* hits = reinterpret_cast<int*>(list + kTopkList);
  uint16_t* gkey = reinterpret_cast<uint16_t*>(hits + kTopkHits);
  __shared__ int4 s_warp[2][kTopkThreads / 32];
  __shared__ int s_hits, s_total, s_list;
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int flip = 0;
  // sums over the block of three values per thread, the same in every thread; one barrier (two sets of slots in turn)
  auto block_sums = [&](int c1, int c2, int c3) {
    c1 = __reduce_add_sync(0xffffffffu, c1);
    c2 = __reduce_add_sync(0xffffffffu, c2);
    c3 = __reduce_add_sync(0xffffffffu, c3);
    if (lane == 0) s_warp[flip][warp] = make_int4(c1, c2, c3, 0);
    __syncthreads();
    int3 s = make_int3(0, 0, 0);
#pragma unroll
    for (int i = 0; i < kTopkThreads / 32; ++i) {
      const int4 w = s_warp[flip][i];
      s.x += w.x;
      s.y += w.y;
      s.z += w.z;
    }
    flip ^= 1;
    return s;
  };
  if (tid == 0) { s_hits = 0; s_total = 0; s_list = 0; }
  __syncthreads();                                       // groups are listed from the first loop on
  pdl_wait();
  pdl_launch_dependents();

  // the window's maxima as ordered 16-bit keys, eight at a time (rows of gmax are 16-byte aligned); whatever else is
  // read from global memory is asked for before the first of them is looked at
  const uint4* g4 = reinterpret_cast<const uint4*>(p.gmax + (size_t)b * p.ld_gmax);
  const int n_vec = (p.n_groups + 7) / 8;
  uint4 raw = tid < n_vec ? __ldcg(&g4[tid]) : make_uint4(0u, 0u, 0u, 0u);
  const unsigned int key_inf = topk_ord16(0xFF80u);      // -inf is never a candidate
  unsigned int kmin = key_inf + 1u;                      // lowest value key a candidate may have
  int held = 0;
  unsigned long long held_key = 0ull;
  if (!p.first) {
    held_key = tid < kTopkMaxK ? p.run[(size_t)b * kTopkMaxK + tid] : 0ull;
    held = p.run_cnt[b];
    kmin = max(kmin, topk_ord16(__float_as_uint(p.thr[b]) >> 16) + 1u);
  }
  auto hit = [&](int g) {
    const int at = atomicAdd(&s_hits, 1);
    if (at < kTopkHits) hits[at] = g;
  };
  unsigned int mine = 0u;                                // the largest of this thread's keys
  for (int i = tid; i < n_vec; i += kTopkThreads) {
    if (i != tid) raw = __ldcg(&g4[i]);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const unsigned int lo = 8 * i + 2 * e < p.n_groups ? topk_ord16(w[e] & 0xFFFFu) : 0u;
      const unsigned int hi = 8 * i + 2 * e + 1 < p.n_groups ? topk_ord16(w[e] >> 16) : 0u;
      mine = max(mine, max(lo, hi));
      if (!p.first && lo >= kmin) hit(8 * i + 2 * e);
      if (!p.first && hi >= kmin) hit(8 * i + 2 * e + 1);
      o[e] = lo | (hi << 16);
    }
    reinterpret_cast<uint4*>(gkey)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  __syncthreads();
  if (p.first || s_hits > 2 * p.k) {
    // Many groups: raise the bound to a key that k of the maxima reach.  With twice as many threads at work as that,
    // the k-th largest of the threads' own maxima will do (a thread has 8 or 16 keys: about a quarter more groups
    // reach it than the exact bound, and a round looks at one key per thread); else of all.  Two bits a round.
    const bool by_thread = min(n_vec, kTopkThreads) >= 2 * p.k;
    unsigned int t = 0u;
    for (int sh = 14; sh >= 0; sh -= 2) {
      const unsigned int t1 = t | (1u << sh), t2 = t | (2u << sh), t3 = t | (3u << sh);
      int n1 = 0, n2 = 0, n3 = 0;
      if (by_thread) {
        n1 = mine >= t1;
        n2 = mine >= t2;
        n3 = mine >= t3;
      } else {
        for (int i = tid; i < n_vec; i += kTopkThreads) {              // (the keys that fill up the last eight are 0)
          raw = reinterpret_cast<const uint4*>(gkey)[i];
          const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const unsigned int g = e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xFFFFu;
            n1 += g >= t1;
            n2 += g >= t2;
            n3 += g >= t3;
          }
        }
      }
      const int3 m = block_sums(n1, n2, n3);
      t = m.z >= p.k ? t3 : m.y >= p.k ? t2 : m.x >= p.k ? t1 : t;
    }
    kmin = max(kmin, t);
    if (tid == 0) s_hits = 0;
    __syncthreads();
    for (int i = tid; i < n_vec; i += kTopkThreads) {
      raw = reinterpret_cast<const uint4*>(gkey)[i];
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if ((e & 1 ? w[e >> 1] >> 16 : w[e >> 1] & 0xFFFFu) >= kmin) hit(8 * i + e);
    }
    __syncthreads();
  }
  const int hit_total = s_hits;
  const bool listed = hit_total <= kTopkHits;
  // every candidate: what is held already, then four threads per group, eight logits each
  auto for_each_global = [&](auto&& f) {
    if (tid < held) f(held_key);
    for (int i = tid >> 2; i < (listed ? hit_total : p.n_groups); i += kTopkThreads / 4) {
      const int g = listed ? hits[i] : i;
      if (gkey[g] < kmin) continue;
      const int chunk = (p.first_group + g) / p.chunk_groups;
      const int id0 = (int)(p.label0 + (long long)chunk * p.chunk_rows) + 32 * (p.first_group + g - chunk * p.chunk_groups) + 8 * (tid & 3);
      const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(p.z + (size_t)b * p.ld_z + 32 * (long long)g + 8 * (tid & 3)));
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t h = e & 1 ? w[e >> 1] & 0xFFFF0000u : w[e >> 1] << 16;
        const float v = __uint_as_float(h);
        if (v == v && topk_ord16(h >> 16) >= kmin) f(topk_key64(v, id0 + e));
      }
    }
  };
  for_each_global([&](unsigned long long key) {
    const int at = atomicAdd(&s_total, 1);
    if (at < kTopkCand) cand[at] = key;
  });
  __syncthreads();
  const int total = s_total;
  const bool in_smem = total <= kTopkCand;
  auto for_each = [&](auto&& f) {
    if (in_smem) {
      for (int i = tid; i < total; i += kTopkThreads) f(cand[i]);
    } else {
      for_each_global(f);
    }
  };
  const unsigned long long* keys = cand;
  int n = total;
  if (total > kTopkList) {
    // the k-th largest value, two bits a round (the low 16 bits of a value follow from its sign)
    unsigned long long kth = 0ull;
    int at_least = total;
    auto search = [&](int first, int last) {
      for (int sh = first; sh >= last; sh -= 2) {
        const unsigned long long t1 = kth | (1ull << sh), t2 = kth | (2ull << sh), t3 = kth | (3ull << sh);
        int n1 = 0, n2 = 0, n3 = 0;
        for_each([&](unsigned long long key) {
          n1 += key >= t1;
          n2 += key >= t2;
          n3 += key >= t3;
        });
        const int3 m = block_sums(n1, n2, n3);
        if (m.z >= p.k) { kth = t3; at_least = m.z; }
        else if (m.y >= p.k) { kth = t2; at_least = m.y; }
        else if (m.x >= p.k) { kth = t1; at_least = m.x; }
      }
    };
    search(62, 48);
    if (at_least > kTopkList) search(46, 0);             // many equal values: go on into the labels
    for_each([&](unsigned long long key) {
      if (key >= kth) {
        const int at = atomicAdd(&s_list, 1);
        if (at < kTopkList) list[at] = key;
      }
    });
    __syncthreads();
    keys = list;
    n = min(s_list, kTopkList);
  }
  // rank by counting
  for (int i = tid; i < n; i += kTopkThreads) {
    const unsigned long long key = keys[i];
    int rank = 0;
    for (int t = 0; t < n; ++t) rank += keys[t] > key;
    if (rank >= p.k) continue;
    const float v = topk_value(key);
    if (p.last) {
      p.out_val[(size_t)b * p.k + rank] = v;
      p.out_idx[(size_t)b * p.k + rank] = (int)(0xFFFFFFFFu - (unsigned int)key);
    } else {
      p.run[(size_t)b * kTopkMaxK + rank] = key;
      if (rank == p.k - 1) p.thr[b] = v;
    }
  }
  if (p.last) {
    for (int i = n + tid; i < p.k; i += kTopkThreads) {   // fewer labels than wanted
      p.out_val[(size_t)b * p.k + i] = -INFINITY;
      p.out_idx[(size_t)b * p.k + i] = -1;
    }
  } else if (tid == 0) {
    p.run_cnt[b] = min(n, p.k);
    if (n < p.k) p.thr[b] = -INFINITY;
  }
}

}  // namespace xmc
