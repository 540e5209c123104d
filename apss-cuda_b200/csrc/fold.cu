// Folded-bound join: row order, folded operands, the choice of widths from
// sampled rows, and the host side of the join (see fold.cuh).
#include <cuda_runtime.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "fold.cuh"
#include "prims.cuh"

namespace cuapss {

namespace {

constexpr int kThreads = 256;
constexpr int kClasses = kFoldClasses;
// Upper edges of the classes as shares of the sorted rows: finer towards the
// long rows, whose folded products spread the most.
constexpr double kClassEdge[kClasses] = {0.125, 0.25, 0.375, 0.5,  0.625, 0.75,  0.8125, 0.875,
                                         0.92,  0.95, 0.97,  0.98, 0.988, 0.994, 0.998,  1.0};
// Joins of fewer 128 x 128 tiles keep the caller's order and one width,
// unsampled, and take at most kSmallMaxCand candidates (small_limit).
constexpr double kSampleMinTiles = 2048.0;
constexpr int kSmallLevel = 3;
constexpr int64_t kSmallMaxCand = 1 << 21;

// Cost model, SM-nanoseconds, measured on 200,000 and 400,000 rows of the
// d = 50,000 workload. A 256 x 128 tile whose I chunks stay resident takes
// kTileNs + kChunkNs per 64 columns and at least kTileMinNs (K = 64: 613, 128:
// 709, 256: 1,371), a streamed one kStreamNs per 64 columns (K = 384: 2,441,
// 1,024: 6,768). A candidate takes kCandNs (its listing in the tile kernel,
// and verify) + kCandEntryNs per entry of its longer row.
constexpr double kTileNs = 55.0, kChunkNs = 328.0, kTileMinNs = 610.0, kStreamNs = 415.0;
constexpr double kCandNs = 45.0, kCandEntryNs = 0.3;
// The probing path's launches and round trips, and its preprocessing per
// non-zero, that a folded join does without (500 .. 8,000 rows of 20 .. 800
// entries in both precisions, few candidates: 0.57-0.70 -> 0.20-0.22 ms at 500
// rows, 0.92 -> 0.23 at 8,000 of 40, 3.8 -> 0.5 of 400; 76 ms of preprocessing
// for 120M non-zeros). An index query prepares nothing but its own rows; a
// batch, whose probing path plans no rare features, about 0.1 ns (400
// instances, 16M non-zeros: 3.1-3.7 ms in all).
constexpr double kProbeFixedNs = 350e3, kProbeEntryNs = 0.6, kBatchProbeEntryNs = 0.1;
// Without length classes a candidate costs kMeanCandNs + kMeanCandEntryNs per
// entry of a row (2,000 rows where all pairs pass: 67 SM-ns at 75 entries, 160 at
// 200, 325 at 400, 655 at 800); where few pass, theirs are the longer rows
// (120 entries in the mean: 102 SM-ns where 0.6 of the pairs pass, 222 where
// 0.02 to 0.08 do).
constexpr double kMeanCandNs = 10.0, kMeanCandEntryNs = 0.8;
double cand_ns(double len, double share) {
  return kMeanCandNs + kMeanCandEntryNs * len * (2.0 - std::min(1.0, share));
}
// Folding a row at a width, per entry and per column.
constexpr double kFoldEntryNs = 0.35, kFoldColumnNs = 0.05;
// FP32, 128 x 128 tiles.
constexpr double kTile32Ns = 380.0, kColumn32Ns = 92.0;

// Joins of at least this long look for tiles too short for one another.
constexpr double kReachMinNs = 500e3;

template <bool MIXED>
constexpr int kPair = MIXED ? 2 : 1;  // I blocks of a tile
template <bool MIXED>
constexpr int kChunk = MIXED ? kFoldChunk16 : kFoldChunk32;

template <bool MIXED>
double tile_cost(int level) {
  const int K = fold_k(MIXED, level);
  if (!MIXED) return kTile32Ns + kColumn32Ns * K;
  return K <= kFoldResident16 ? std::max(kTileMinNs, kTileNs + kChunkNs * (K / 64))
                              : kStreamNs * (K / 64);
}

template <bool MIXED>
cuapss_status launch_fold(const FoldTileArgs& a, int sms, cudaStream_t st, bool count) {
  return MIXED ? launch_tiles_fold(a, sms, st, count) : launch_tiles_fold32(a, sms, st, count);
}

inline unsigned grid_for(int64_t work, int per_block) {
  const int64_t g = ceil_div(std::max<int64_t>(work, 1), per_block);
  return (unsigned)std::min<int64_t>(g, 148 * 32);
}

constexpr float kSquareScale = 2147483648.0f;  // 2^31, of fixed-point squares

// ---- row order: by length, in 256 classes of about 1/16 octave -----------
// Rows with thresholds of their own are ordered by length over the squared
// room between t and the usual product of unrelated rows: both make folded
// products pass.
__global__ void k_len_keys(const int64_t* __restrict__ rp, const float* __restrict__ t_row,
                           int64_t n, uint64_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float len = (float)(rp[i + 1] - rp[i]);
    if (t_row) {
      const float room = fmaxf(t_row[i] - 0.15f, 0.1f);
      len *= 0.1f / (room * room);
    }
    keys[i] = (uint64_t)min(255, (int)(16.0f * __log2f(fmaxf(len, 1.0f))));
    vals[i] = (uint32_t)i;
  }
}

__global__ void k_order(const uint32_t* __restrict__ sorted, int64_t n, int64_t slots,
                        int32_t* __restrict__ rowmap) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < slots;
       i += (int64_t)gridDim.x * blockDim.x)
    rowmap[i] = i < n ? (sorted ? (int32_t)sorted[i] : (int32_t)i) : -1;
}

// ---- batches: each instance's rows from a block boundary on ---------------
// tab[4 q ..] = {first place, first row, rows, threshold bits} of instance q;
// places past its rows up to the next block boundary are empty.
__global__ void k_batch_places(const int64_t* __restrict__ tab, int k, int32_t* __restrict__ rowmap,
                               float* __restrict__ t_place) {
  for (int q = blockIdx.x; q < k; q += gridDim.x) {
    const int64_t S = tab[4 * q], R = tab[4 * q + 1], n = tab[4 * q + 2];
    const float t = __int_as_float((int)tab[4 * q + 3]);
    const int64_t npad = (n + kBlockRows - 1) / kBlockRows * kBlockRows;
    for (int64_t r = threadIdx.x; r < npad; r += blockDim.x) {
      rowmap[S + r] = r < n ? (int32_t)(R + r) : -1;
      t_place[S + r] = t;
    }
  }
}

// ---- rows too short for one another ---------------------------------------
// A row with k entries shares at most k features with row b, so their product
// is at most the first one's norm times the norm of b's k largest entries:
// below need(b) = the k at which that reaches t, the pair cannot be in the
// answer. One warp per place finds a lower bound of need(b): for a cut c, with
// S and n the sum and number of b's squares above c and S < T = (t / norm)^2,
// need >= n + (T - S) / c. Each block gets its smallest need and its longest
// row.
constexpr int kNeedRegs = 4;  // entries a lane keeps in registers
__global__ void k_block_needs(const int32_t* __restrict__ rowmap, int64_t slots,
                              const int64_t* __restrict__ rp, const float* __restrict__ val,
                              uint32_t T, int* __restrict__ need, int* __restrict__ longest) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t s = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; s < slots; s += warps) {
    const int32_t r = rowmap[s];
    if (r < 0) continue;  // warp-uniform
    const int64_t lo = rp[r];
    const int len = (int)(rp[r + 1] - lo);
    // squares in multiples of 2^-31, rounded up: sums of them are exact
    uint32_t q[kNeedRegs];
    auto square = [&](int e) {
      const float v = val[lo + e];
      return __float2uint_ru(__fmul_ru(v, v) * kSquareScale);
    };
    uint32_t top = 0;
#pragma unroll
    for (int k = 0; k < kNeedRegs; ++k) {
      q[k] = lane + 32 * k < len ? square(lane + 32 * k) : 0u;
      top = max(top, q[k]);
    }
    for (int e = lane + 32 * kNeedRegs; e < len; e += 32) top = max(top, square(e));
    top = __reduce_max_sync(0xffffffffu, top);
    // the largest cut (of eight halvings) whose sum above stays below T gives
    // the bound; the cut at the top has nothing above it
    uint32_t below = 0, above = top;  // sums: >= T at `below` or not known, < T at `above`
    uint32_t S = 0;
    int n = 0;
    for (int it = 0; it < 8; ++it) {
      const uint32_t c = below + (above - below) / 2;
      uint32_t sum = 0;
      int cnt = 0;
#pragma unroll
      for (int k = 0; k < kNeedRegs; ++k)
        if (q[k] > c) {
          sum += q[k];
          ++cnt;
        }
      for (int e = lane + 32 * kNeedRegs; e < len; e += 32) {
        const uint32_t x = square(e);
        if (x > c) {
          sum += x;
          ++cnt;
        }
      }
      sum = __reduce_add_sync(0xffffffffu, sum);
      cnt = __reduce_add_sync(0xffffffffu, cnt);
      if (sum < T) {
        above = c;
        S = sum;
        n = cnt;
      } else {
        below = c;
      }
    }
    if (lane == 0) {
      const uint32_t c = max(above, 1u);
      const int k = min(len, n + (int)min((T - S) / c, 0x3fffffffu));
      atomicMin(&need[s / kBlockRows], k);
      atomicMax(&longest[s / kBlockRows], len);
    }
  }
}

// ---- sampled rows: up to 128 of each class, evenly spaced ----------------
struct ClassRows {
  int64_t row[kClasses + 1];  // first row of each class, n at the end
};

__global__ void k_sample_rows(const int32_t* __restrict__ rowmap, const int64_t* __restrict__ rp,
                              ClassRows C, int32_t* __restrict__ sample,
                              unsigned long long* __restrict__ len_sum) {
  const int c = blockIdx.x, k = threadIdx.x;
  const int64_t lo = C.row[c], m = C.row[c + 1] - lo;
  int32_t r = -1;
  if (m >= kBlockRows) r = rowmap[lo + (int64_t)k * m / kBlockRows];
  else if (k < m) r = rowmap[lo + k];
  sample[c * kBlockRows + k] = r;
  if (r >= 0) atomicAdd(&len_sum[c], (unsigned long long)(rp[r + 1] - rp[r]));
}

// ---- folded rows ---------------------------------------------------------
// A row's entries are summed per column of every wanted width in shared
// memory, in one pass over the row, and written as BF16 in the
// 128-byte-swizzled chunk layout of the tensor cores (prep.cu), or as FP32.
// Shared columns sum the squares, each rounded up to a multiple of 2^-31, as
// integers (a row's squared norm is below 1.9; integer shared-memory atomics
// run at 12 a clock and SM against 3.4 for FP32: 200,000 rows of the d = 1M
// workload, 619 -> 394 us together with leaving out the widths that do not
// pay), and every step from there on rounds up, so their products bound the
// exact ones. Head values are rounded to nearest, which the margin covers, or
// up where no value is negative: no margin is then needed for them (it costs
// 4% of the tile time at t = 0.5).
__host__ __device__ constexpr size_t fold_bytes(bool mixed, int level) {  // of a row block
  return (size_t)fold_k(mixed, level) * kBlockRows * (mixed ? 2 : 4);
}

// First accumulator column of level l when the levels of `mask` lie one
// after another, and their total.
__host__ __device__ constexpr int fold_offset(bool mixed, uint32_t mask, int l) {
  int o = 0;
  for (int k = 0; k < l; ++k)
    if ((mask >> k) & 1u) o += fold_k(mixed, k);
  return o;
}

// Bytes of a row block's levels below l.
constexpr size_t fold_offset_bytes(bool mixed, int l) {
  size_t o = 0;
  for (int k = 0; k < l; ++k) o += fold_bytes(mixed, k);
  return o;
}

// A level's columns, for loops over the levels of a mask: k columns, p of them
// exact, m = k - p shared; x / m = umulhi(x, magic) >> shift for x < 2^31
// (magic = ceil(2^(31 + s) / m) with s = ceil(log2 m): the error x e / (m
// 2^(31 + s)), e < m <= 2^s, is below 1 / m).
struct FoldDiv {
  uint32_t k, p, m, magic, shift;
};
struct FoldDivs {
  FoldDiv d[2][kFoldLevels];
};
constexpr FoldDivs fold_divs() {
  FoldDivs t{};
  for (int f = 0; f < 2; ++f)
    for (int l = 0; l < kFoldLevels; ++l) {
      const uint32_t k = (uint32_t)fold_k(f == 1, l), m = k - k / 4;
      uint32_t s = 0;
      while ((1u << s) < m) ++s;
      const uint64_t pow = 1ull << (31 + s);
      t.d[f][l] = {k, k / 4, m, (uint32_t)((pow + m - 1) / m), s - 1};
    }
  return t;
}
__constant__ const FoldDivs kFoldDivs = fold_divs();

// Runs f(l, D) for the levels l of mask (the row's threads take the same
// branches): unrolled, with constants for D, or as a loop.
template <bool MIXED, bool UNROLL, typename F>
__device__ __forceinline__ void fold_for_levels(uint32_t mask, F&& f) {
  if constexpr (UNROLL) {
#pragma unroll
    for (int l = 0; l < kFoldLevels; ++l)
      if ((mask >> l) & 1u) {
        const uint32_t k = (uint32_t)fold_k(MIXED, l);
        f(l, FoldDiv{k, k / 4, k - k / 4, 0, 0});
      }
  } else {
    for (uint32_t w = mask; w; w &= w - 1) {
      const int l = __ffs(w) - 1;
      f(l, kFoldDivs.d[MIXED][l]);
    }
  }
}

// N entries of a row into the columns of every level of mask (f: rank, < 0:
// none).
template <bool MIXED, int N, bool UNROLL>
__device__ __forceinline__ void fold_add(uint32_t mask, uint32_t* acc, const int32_t (&f)[N],
                                         const float (&v)[N]) {
  uint32_t square[N];
#pragma unroll
  for (int q = 0; q < N; ++q) square[q] = __float2uint_ru(__fmul_ru(v[q], v[q]) * kSquareScale);
  fold_for_levels<MIXED, UNROLL>(mask, [&](int, const FoldDiv D) {
#pragma unroll
    for (int q = 0; q < N; ++q) {
      const uint32_t r = (uint32_t)f[q], x = r - D.p;
      if (r < D.p) acc[r] = __float_as_uint(v[q]);
      else if (f[q] >= 0)
        atomicAdd(&acc[D.p + (UNROLL ? x % D.m : x - (__umulhi(x, D.magic) >> D.shift) * D.m)],
                  square[q]);
    }
    acc += D.k;
  });
}

// Norm of a shared column from its fixed-point squares, times scale: an upper
// bound (sqrt.approx is within 2^-23 of the root; scale carries a factor
// 1 + 2^-21 for it). The IEEE root and the software round-up conversion to
// BF16 took most of the instructions of folding short rows (1.6M rows of 30:
// 1,348 -> 961 us; 200,000 rows of 120: 394 -> 301 us).
__device__ __forceinline__ float fold_norm(uint32_t squares, float scale) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(__uint2float_ru(squares) * (1.0f / kSquareScale)));
  return __fmul_ru(r, scale);
}

// Two non-negative floats rounded up to BF16, packed.
__device__ __forceinline__ uint32_t bf16x2_up(float lo, float hi) {
  return __byte_perm(__float_as_uint(lo) + 0xffffu, __float_as_uint(hi) + 0xffffu, 0x7632);
}

// A row's sums to its place (block b, row rr) in every level of mask.
template <bool MIXED, bool UNROLL>
__device__ __forceinline__ void fold_write(uint32_t mask, const uint32_t* acc, const FoldOut& O,
                                           float scale, bool nonneg, int b, int rr, int tid,
                                           int nt) {
  const float up = __fmul_ru(scale, 1.0f + 4.76837158e-7f);  // 1 + 2^-21
  fold_for_levels<MIXED, UNROLL>(mask, [&](int l, const FoldDiv D) {
    const int K = (int)D.k, P = K / 4;
    const uint32_t* a = acc;
    acc += K;
    uint8_t* dst = O.base[l] + (size_t)(b - O.first[l]) * ((size_t)K * kBlockRows * (MIXED ? 2 : 4));
    if (!MIXED) {  // [column][row]
      for (int c = tid; c < K; c += nt)
        reinterpret_cast<float*>(dst)[c * kBlockRows + rr] =
            c < P ? __uint_as_float(a[c]) * scale : fold_norm(a[c], up);
      return;
    }
    uint4* out = reinterpret_cast<uint4*>(dst);
    for (int c8 = tid; c8 < K / 8; c8 += nt) {
      const uint4 x = reinterpret_cast<const uint4*>(a)[2 * c8];
      const uint4 y = reinterpret_cast<const uint4*>(a)[2 * c8 + 1];
      const uint32_t f[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (c8 * 8 >= P) {  // P is a multiple of 8
          w[q] = bf16x2_up(fold_norm(f[2 * q], up), fold_norm(f[2 * q + 1], up));
        } else if (nonneg) {
          w[q] = bf16x2_up(__fmul_ru(__uint_as_float(f[2 * q]), scale),
                           __fmul_ru(__uint_as_float(f[2 * q + 1]), scale));
        } else {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(f[2 * q]) * scale,
                                                         __uint_as_float(f[2 * q + 1]) * scale);
          memcpy(&w[q], &h, 4);
        }
      }
      const int kc = c8 >> 3, c = c8 & 7;
      out[((size_t)kc * kBlockRows + rr) * 8 + (c ^ (rr & 7))] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  });
}

// t_row (per caller's row, may be null): the row is folded divided by its
// threshold, so that one threshold of 1 serves rows of different ones.
// GROUP threads per row (8 .. 32, or the whole CTA for long rows). Blocks
// [b0, b1) of rowmap; blk_mask[b]: levels of block b (null: mask0 for all);
// only blocks with (wide) or without a level that is not narrow are taken.
// Bound by instructions: 425 a row of 30 entries in 192 columns when every
// entry went through ten unrolled level tests with their offsets; a loop over
// the levels that the block has, 4 entries at a time, 8 threads a row, takes
// 1,112 -> 594 us for 1.6M such rows (672 with the unrolled tests). Longer
// rows keep the unrolled levels, whose divisions are constants, and take
// several entries between the tests: 200,000 rows of 120, a warp each, 308 ->
// 275 us; rows with wide levels 143 -> 130 us (170 as a loop).
// Shared memory: max_col columns per row, the most that a block's levels
// have.
constexpr uint32_t kNarrowLevels = 0x7f;  // K <= 512 (mixed), 192 (FP32)

template <bool MIXED, int GROUP>
__global__ void __launch_bounds__(kThreads)
    k_fold_rows(const int32_t* __restrict__ rowmap, int64_t slot0, int64_t slot1,
                const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                const float* __restrict__ val, const int32_t* __restrict__ perm,
                const float* __restrict__ t_row, bool nonneg,
                const uint16_t* __restrict__ blk_mask, uint32_t mask0, int max_col, bool wide,
                const __grid_constant__ FoldOut O) {
  extern __shared__ __align__(16) uint32_t fold_sm[];
  constexpr int kGroups = kThreads / GROUP;
  constexpr bool kUnroll = GROUP >= 32;
  constexpr int N = GROUP > 32 ? 2 : 4;
  const int tid = threadIdx.x % GROUP;
  uint32_t* acc = fold_sm + (threadIdx.x / GROUP) * max_col;
  for (int64_t s = slot0 + (int64_t)blockIdx.x * kGroups + threadIdx.x / GROUP; s < slot1;
       s += (int64_t)gridDim.x * kGroups) {
    const int b = (int)(s / kBlockRows), rr = (int)(s % kBlockRows);
    const uint32_t mask = blk_mask ? (uint32_t)blk_mask[b] : mask0;
    if (mask == 0 || ((mask & ~kNarrowLevels) != 0) != wide) continue;  // same for the warp
    const int ncol = fold_offset(MIXED, mask, kFoldLevels);
    const int32_t r = rowmap[s];
    const int64_t lo = r >= 0 ? rp[r] : 0;
    const int len = r >= 0 ? (int)(rp[r + 1] - lo) : 0;
    for (int k = tid; k < ncol / 4; k += GROUP)
      reinterpret_cast<uint4*>(acc)[k] = make_uint4(0u, 0u, 0u, 0u);
    if (GROUP <= 32) __syncwarp();
    else __syncthreads();
    for (int e0 = 0; e0 < len; e0 += N * GROUP) {
      int32_t f[N];
      float v[N];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int e = e0 + q * GROUP + tid;
        f[q] = e < len ? perm[col[lo + e]] : -1;
        v[q] = e < len ? val[lo + e] : 0.0f;
      }
      fold_add<MIXED, N, kUnroll>(mask, acc, f, v);
    }
    if (GROUP <= 32) __syncwarp();
    else __syncthreads();
    const float scale = t_row && r >= 0 ? __frcp_ru(t_row[r]) : 1.0f;
    fold_write<MIXED, kUnroll>(mask, acc, O, scale, nonneg, b, rr, tid, GROUP);
    if (GROUP <= 32) __syncwarp();
    else __syncthreads();
  }
}

// Threads per row. Short rows leave most of a warp idle, in their entries (30)
// and in writing 64 columns (8 lanes): 8 or 16 threads take a row where its
// columns leave room for the CTA's rows in shared memory (8 rows a warp of
// 512 columns: 64 KB a CTA) and the rows fill 8 CTAs a SM (20,000 rows: 54 us
// with 8 threads a row, 24 with 16, 30 with 32).
constexpr int kFoldCols8 = 512;
constexpr int64_t kFoldRows8 = 148 * 8 * (kThreads / 8);
constexpr int kFoldSmem = 64 * 1024;
static_assert(fold_offset(true, kNarrowLevels, kFoldLevels) * 8 * 4 <= kFoldSmem &&
                  fold_offset(false, kNarrowLevels, kFoldLevels) * 8 * 4 <= kFoldSmem &&
                  fold_offset(true, (1u << kFoldLevels) - 1, kFoldLevels) * 4 <= kFoldSmem &&
                  fold_offset(false, (1u << kFoldLevels) - 1, kFoldLevels) * 4 <= kFoldSmem &&
                  kFoldCols8 * (kThreads / 8) * 4 <= kFoldSmem,
              "shared memory of folded rows");

// Folds the places of [0, slots) with the levels of masks (host, per block;
// empty: mask0 everywhere) into O.
template <bool MIXED>
cuapss_status fold_places(const FoldSide& s, const int32_t* rowmap, int64_t slots,
                          const std::vector<uint16_t>& masks, uint32_t mask0, const int32_t* perm,
                          const FoldOut& O, Workspace& ws, const std::string& tag,
                          cudaStream_t st) {
  uint16_t* d_mask = nullptr;
  // most columns of a block, and blocks, without and with a wide level
  int cols[2] = {0, 0};
  int64_t b0[2] = {0, 0}, b1[2] = {0, 0};
  if (masks.empty()) {
    const int w = (mask0 & ~kNarrowLevels) ? 1 : 0;
    cols[w] = fold_offset(MIXED, mask0, kFoldLevels);
    b1[w] = slots / kBlockRows;
  } else {
    ST_TRY(ws.get(tag + ":mask", masks.size(), &d_mask));
    CU_TRY(cudaMemcpyAsync(d_mask, masks.data(), 2 * masks.size(), cudaMemcpyHostToDevice, st));
    for (size_t b = 0; b < masks.size(); ++b) {
      if (!masks[b]) continue;
      const int w = (masks[b] & ~kNarrowLevels) ? 1 : 0;
      if (!cols[w]) b0[w] = (int64_t)b;
      cols[w] = std::max(cols[w], fold_offset(MIXED, masks[b], kFoldLevels));
      b1[w] = (int64_t)b + 1;
    }
  }
  const DevCsr& x = s.x;
  for (int w = 0; w < 2; ++w) {
    if (!cols[w]) continue;
    const int64_t rows = (b1[w] - b0[w]) * kBlockRows;
    auto run = [&](auto kernel, int group) -> cuapss_status {
      const size_t smem = (size_t)cols[w] * 4 * (kThreads / group);
      CU_TRY(cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kFoldSmem));
      kernel<<<grid_for(rows, kThreads / group), kThreads, smem, st>>>(
          rowmap, b0[w] * kBlockRows, b1[w] * kBlockRows, x.rp, x.col, x.val, perm, s.t_row,
          x.nonneg, d_mask, mask0, cols[w], w == 1, O);
      LAUNCH_CHECK();
      return CUAPSS_OK;
    };
    if (w == 1) ST_TRY(run(k_fold_rows<MIXED, kThreads>, kThreads));  // and the samples
    else if (cols[w] <= kFoldCols8 && rows >= kFoldRows8) ST_TRY(run(k_fold_rows<MIXED, 8>, 8));
    else if (cols[w] <= 2 * kFoldCols8 && rows >= kFoldRows8 / 2)
      ST_TRY(run(k_fold_rows<MIXED, 16>, 16));
    else ST_TRY(run(k_fold_rows<MIXED, 32>, 32));
  }
  return CUAPSS_OK;
}

// Margin of the bound of a level's products, for rows folded as they are
// (t_min = 1: thresholds compare directly) or divided by thresholds of at
// least t_min.
float fold_eps(bool mixed, int level, double nrm2, double t_min, bool nonnegI, bool nonnegJ) {
  // mixed: BF16 rounding of the head columns (to nearest 2^-8, up 2^-7; up on
  // both sides only raises the product), FP32 accumulation of K / 16 steps;
  // FP32: a chain of K FMAs
  const int K = fold_k(mixed, level);
  const double eI = std::ldexp(1.0, nonnegI ? -7 : -8), eJ = std::ldexp(1.0, nonnegJ ? -7 : -8);
  const double head = !mixed || (nonnegI && nonnegJ) ? 0.0 : eI + eJ + eI * eJ;
  const double acc =
      (mixed ? (K / 16.0 + 2.0) * std::ldexp(1.0, -20) : (K + 4.0) * std::ldexp(1.0, -24)) * 1.02;
  return (float)(((head + acc) * nrm2 * 1.001 + 1e-6) / t_min);
}

// Row order (by length, or as given) and class edges.
cuapss_status order_side(FoldSide& s, bool by_length, const FoldAlloc& alloc, Workspace& ws,
                         const std::string& tag, cudaStream_t st) {
  s.nb = (int)ceil_div(s.x.n, kBlockRows);
  const int64_t slots = (int64_t)s.nb * kBlockRows;
  void* map = nullptr;
  ST_TRY(alloc("map", (size_t)slots * 4, &map));
  s.rowmap = static_cast<int32_t*>(map);
  uint32_t* vals = nullptr;
  if (by_length) {
    uint64_t* keys = nullptr;
    ST_TRY(ws.get(tag + ":keys", (size_t)s.x.n, &keys));
    ST_TRY(ws.get(tag + ":vals", (size_t)s.x.n, &vals));
    k_len_keys<<<grid_for(s.x.n, kThreads), kThreads, 0, st>>>(s.x.rp, s.t_row, s.x.n, keys, vals);
    LAUNCH_CHECK();
    ST_TRY(radix_sort_pairs(keys, vals, s.x.n, 8, ws, tag, st));
  }
  k_order<<<grid_for(slots, kThreads), kThreads, 0, st>>>(vals, s.x.n, slots, s.rowmap);
  LAUNCH_CHECK();
  for (int c = 0; c < kClasses; ++c)
    s.edge[c + 1] = c + 1 == kClasses ? s.nb : std::min(s.nb, (int)(kClassEdge[c] * s.nb) & ~1);
  return CUAPSS_OK;
}

ClassRows class_rows(const FoldSide& s) {
  ClassRows c;
  for (int k = 0; k <= kClasses; ++k)
    c.row[k] = std::min<int64_t>(s.x.n, (int64_t)s.edge[k] * kBlockRows);
  return c;
}

constexpr int64_t kSampleSlots = (int64_t)kClasses * kBlockRows;

// Samples a side's classes and folds the samples at every level of `levels`.
// len_sum (device, kClasses words, zeroed) receives the sampled rows' lengths.
template <bool MIXED>
cuapss_status sample_side(FoldSide& s, uint32_t levels, unsigned long long* len_sum,
                          const int32_t* perm, const FoldAlloc& alloc, Workspace& ws,
                          const std::string& tag, cudaStream_t st) {
  void* p = nullptr;
  ST_TRY(alloc("sample", (size_t)kSampleSlots * 4, &p));
  s.sample = static_cast<int32_t*>(p);
  k_sample_rows<<<kClasses, kBlockRows, 0, st>>>(s.rowmap, s.x.rp, class_rows(s), s.sample,
                                                 len_sum);
  LAUNCH_CHECK();
  size_t total = 0;
  for (int l = 0; l < kFoldLevels; ++l)
    if ((levels >> l) & 1u) total += kClasses * fold_bytes(MIXED, l);
  ST_TRY(alloc("samples", total, &p));
  uint8_t* at = static_cast<uint8_t*>(p);
  for (int l = 0; l < kFoldLevels; ++l) {
    if (!((levels >> l) & 1u)) continue;
    s.sample_out.base[l] = at;
    at += kClasses * fold_bytes(MIXED, l);
  }
  return fold_places<MIXED>(s, s.sample, kSampleSlots, {}, levels, perm, s.sample_out, ws, tag, st);
}

// One join of two sides (or of a side with itself) through the tile kernel.
struct FoldTask {
  FoldSide* I = nullptr;
  FoldSide* J = nullptr;
  bool self = false;
  float t = 1.0f;           // threshold of the folded products
  double t_min = 1.0;       // lowest threshold the I rows were divided by
  int64_t j_offset = 0;     // added to the J row of every pair
  int level[kClasses][kClasses] = {};  // width of each pair of classes
  double cost = 0.0, cands = 0.0;      // modelled SM-nanoseconds, expected candidates
  // self-joins: the last J block whose rows can match rows as short as those
  // of each I block (empty: all)
  std::vector<int> last;
  std::vector<int4> units;
  int64_t tiles = 0;
  int4* d_units = nullptr;
  int64_t cap = 0;
  int64_t limit = 0;  // > 0: with more candidates the probing path is faster
  // Adds the 128 x 128 tiles that the units multiply, by width.
  void count_tiles(int pair, int64_t* tiles_of) const {
    for (const int4& u : units) {
      const bool one = pair == 1 || u.x + 1 >= I->nb || (u.w & kFoldSingle) != 0;
      int64_t n = (int64_t)(u.z - u.y) * (one ? 1 : 2);
      if (self && !one && u.y == u.x) --n;  // block I + 1 starts at itself
      tiles_of[u.w & 0x7f] += n;
    }
  }
};

// Whether a level is sampled for a pair of classes: the widest ones only pay
// where both rows are long (all of them for all pairs took 212 us of a 1.5 ms
// FP32 join of 20,000 rows).
bool sampled_level(int l, int a, int b) {
  const int lo = std::min(a, b), sum = a + b;
  return l < 7 || (l == 7 && sum >= 10) || (l == 8 && sum >= 16) || (l == 9 && lo >= 9);
}

// The levels worth sampling when a sampled tile may take at_most_ns (an FP32
// tile of 1,024 columns takes 190 us beside another).
template <bool MIXED>
uint32_t sampled_levels(double at_most_ns) {
  uint32_t all = (1u << kFoldLevels) - 1u;
  for (int l = kSmallLevel + 1; l < kFoldLevels; ++l)
    if ((MIXED ? 1.0 : 2.0) * tile_cost<MIXED>(l) > at_most_ns) all &= ~(1u << l);
  return all;
}

// The share of the pairs of unrelated rows of mean length len that a fold of K
// columns lets pass at t: it depends on y = (1 - t) len / K alone, within a
// factor of about three (rows of 20 .. 800 entries, d = 1,000 and 50,000, Zipf
// 0.6 .. 1.1, both precisions, t = 0.3 .. 0.9: at y = 0.08 1e-4, 0.12 2e-3,
// 0.18 0.02, 0.34 0.2, 0.5 0.5).
double passing_share(double len, int K, double t) {
  constexpr double y[] = {0.08, 0.12, 0.18, 0.34, 0.5, 0.8};
  constexpr double s[] = {-4.0, -2.7, -1.7, -0.7, -0.3, 0.0};
  const double x = (1.0 - t) * len / K;
  int k = 1;
  while (k < 5 && x > y[k]) ++k;
  return std::pow(10.0, std::min(0.0, s[k - 1] + (x - y[k - 1]) * (s[k] - s[k - 1]) / (y[k] - y[k - 1])));
}

double mean_len(const DevCsr& x) { return (double)x.nnz / (double)std::max<int64_t>(x.n, 1); }

// The wider levels whose sampled tiles take at most a tenth of the probing
// path's fixed cost, where the long rows (kLongRows times the mean, kLongShare
// of the pairs) have candidates at the next narrower width that cost more than
// sampling another does. (Mixed joins of few thousand rows; 8,320 rows of 75
// entries at t = 0.5 with nothing wider than 256 sampled: 1.47 ms, now 0.44; of
// 30 entries at t = 0.7, where no wider one is useful: 0.35 with all sampled,
// 0.32. FP32 samples and small tiles cost more than the model says: 8,320 rows
// of 120 at t = 0.8 2.05 -> 2.49 ms.)
constexpr double kLongRows = 3.0, kLongShare = 0.06, kWideSampleNs = 20e3;
template <bool MIXED>
uint32_t useful_levels(double len, double t, double pairs, int sms) {
  uint32_t use = sampled_levels<MIXED>(0.1 * kProbeFixedNs);
  for (int l = kSmallLevel + 1; l < kFoldLevels; ++l) {
    const double share = passing_share(kLongRows * len, fold_k(MIXED, l - 1), t);
    if (share * kLongShare * pairs * cand_ns(len, share) < kWideSampleNs * sms) use &= ~(1u << l);
  }
  return use;
}

// The width of every pair of classes, from the products of sampled rows, the
// modelled cost of the join and its expected candidates. Levels the J side
// does not hold (FoldSide::levels) are left out.
template <bool MIXED>
cuapss_status plan_levels(cuapss_ctx* ctx, FoldTask& k, const int32_t* perm, double nrm2) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  FoldSide& I = *k.I;
  FoldSide& J = *k.J;
  const size_t ncnt = (size_t)kFoldLevels * kClasses * kClasses;
  unsigned long long* stats = nullptr;  // row length sums, control words, pair counts
  ST_TRY(ws.get("fold:stats", 2 * kClasses + 1 + ncnt / 2, &stats));
  int* ctl = reinterpret_cast<int*>(stats + 2 * kClasses);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(stats + 2 * kClasses + 1);
  const size_t stat_bytes = 8 * (2 * kClasses + 1) + 4 * ncnt;
  CU_TRY(cudaMemsetAsync(stats, 0, stat_bytes, st));
  uint32_t all = 0;
  for (uint32_t m : J.levels) all |= m;
  // no more than a tenth of a small join
  const double tiles128 = (k.self ? 0.5 : 1.0) * I.nb * J.nb;
  all &= sampled_levels<MIXED>(0.1 * tiles128 / kPair<MIXED> / ctx->sms *
                               tile_cost<MIXED>(kSmallLevel)) |
         (MIXED ? useful_levels<MIXED>(std::max(mean_len(I.x), mean_len(J.x)), k.t * k.t_min,
                                       tiles128 * kBlockRows * kBlockRows, ctx->sms)
                : 0u);
  auto temp = [&](const char* tag) {
    return [&ws, tag](const std::string& name, size_t bytes, void** out) {
      return ws.get(tag + name, bytes, out);
    };
  };
  ST_TRY(sample_side<MIXED>(I, all, stats, perm, temp("fold:sI:"), ws, "fold:sI", st));
  if (!k.self && !J.sample)
    ST_TRY(sample_side<MIXED>(J, all, stats + kClasses, perm, temp("fold:sJ:"), ws, "fold:sJ", st));
  FoldTileArgs ta;
  std::vector<int4> units;
  for (int l = kFoldLevels - 1; l >= 0; --l) {
    if (!((all >> l) & 1u)) continue;
    ta.lev[l].I = I.sample_out.base[l];
    ta.lev[l].J = J.sample_out.base[l];
    ta.lev[l].nkc = fold_k(MIXED, l) / kChunk<MIXED>;
    ta.lev[l].eps = fold_eps(MIXED, l, nrm2, k.t_min, k.I->x.nonneg, k.J->x.nonneg);
    for (int a = 0; a < kClasses; a += kPair<MIXED>) {
      if (I.edge[std::min(kClasses, a + kPair<MIXED>)] == I.edge[a]) continue;  // no rows
      for (int b = k.self ? a : 0; b < kClasses; ++b)
        if (J.edge[b + 1] > J.edge[b] && sampled_level(l, a + kPair<MIXED> - 1, b))
          units.push_back(make_int4(a, b, b + 1, l));
    }
  }
  int4* d_units = nullptr;
  ST_TRY(ws.get("fold:sunits", units.size(), &d_units));
  CU_TRY(cudaMemcpyAsync(d_units, units.data(), sizeof(int4) * units.size(),
                         cudaMemcpyHostToDevice, st));
  ta.nI = ta.nJ = kSampleSlots;
  ta.nbI = ta.nbJ = kClasses;
  ta.t = k.t;
  ta.units = d_units;
  ta.nunits = (int)units.size();
  ta.unit_counter = ctl;
  ta.err = ctl + 1;
  ta.class_count = cnt;
  ST_TRY(launch_fold<MIXED>(ta, ctx->sms, st, true));
  std::vector<unsigned long long> h(stat_bytes / 8);
  CU_TRY(cudaMemcpyAsync(h.data(), stats, stat_bytes, cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  const int herr = (int)(h[2 * kClasses] >> 32);
  if (herr & kErrTimeout) return CUAPSS_ETIMEOUT;
  if (herr) return CUAPSS_ECUDA;
  const uint32_t* hc = reinterpret_cast<const uint32_t*>(h.data() + 2 * kClasses + 1);
  const ClassRows cr[2] = {class_rows(I), class_rows(J)};
  double rows[2][kClasses];
  FoldSide* side[2] = {&I, &J};
  for (int q = 0; q < 2; ++q)
    for (int c = 0; c < kClasses; ++c) {
      rows[q][c] = (double)std::min<int64_t>(kBlockRows, cr[q].row[c + 1] - cr[q].row[c]);
      if (q == 1 && (k.self || J.prepared)) continue;  // known already
      side[q]->len[c] = rows[q][c] > 0 ? (double)h[q * kClasses + c] / rows[q][c] : 0.0;
    }
  // J chunks of a prepared index come from HBM: its bandwidth, an SM's share
  const double load_ns_per_byte = J.prepared ? ctx->sms / 6500.0 : 0.0;
  // cost[l][a][b], share[l][a][b] of every level that was sampled
  const double kNever = 1e300;
  std::vector<double> cost(ncnt, kNever), found(ncnt, 0.0);
  // (a pair of classes' levels side by side for the eleven passes of choose: a
  // 20,000-row join 371 -> 361 us, a 256-row query 482 -> 469 against levels
  // outermost)
  auto at = [](int l, int a, int b) { return ((size_t)a * kClasses + b) * kFoldLevels + l; };
  for (int a = 0; a < kClasses; ++a)
    for (int b = k.self ? a : 0; b < kClasses; ++b) {
      const double sampled = rows[0][a] * rows[1][b] - (k.self && a == b ? rows[0][a] : 0.0);
      const double nI = (double)(cr[0].row[a + 1] - cr[0].row[a]);
      const double nJ = (double)(cr[1].row[b + 1] - cr[1].row[b]);
      const double pairs = k.self && a == b ? nI * (nI - 1) / 2 : nI * nJ;
      if (pairs <= 0) continue;
      const double tiles = k.self ? pairs / ((double)kPair<MIXED> * kBlockRows * kBlockRows)
                                  : std::ceil(nI / (kPair<MIXED> * kBlockRows)) *
                                        std::ceil(nJ / kBlockRows);
      for (int l = 0; l < kFoldLevels; ++l) {
        // (a mixed sample tile spans the classes a, a + 1 of an even a)
        if (!((all & J.levels[b]) >> l & 1u) || !sampled_level(l, a | (kPair<MIXED> - 1), b)) continue;
        double c = (double)hc[((size_t)l * kClasses + a) * kClasses + b];
        if (k.self && a == b) c = std::max(0.0, c - rows[0][a]);  // a row with itself
        // a count of zero is not a share of zero: half a pair
        const double share = sampled > 0 ? std::max(c, 0.5) / sampled : 0.0;
        const double cand_ns = kCandNs + kCandEntryNs * std::max(I.len[a], J.len[b]);
        const double load = (double)fold_bytes(MIXED, l) * load_ns_per_byte;
        found[at(l, a, b)] = share * pairs;
        cost[at(l, a, b)] = tiles * std::max(tile_cost<MIXED>(l), load) + share * pairs * cand_ns;
      }
    }
  // the best level of each pair of classes among `use`, and what folding the
  // rows at the levels taken costs
  auto choose = [&](uint32_t use, bool write) {
    double sum = 0.0;
    uint32_t needI[kClasses] = {}, needJ[kClasses] = {};
    if (write) k.cands = 0.0;
    for (int a = 0; a < kClasses; ++a)
      for (int b = k.self ? a : 0; b < kClasses; ++b) {
        const double* c = &cost[at(0, a, b)];
        int best = -1;
        double least = kNever;
        for (int l = 0; l < kFoldLevels; ++l)
          if (((use >> l) & 1u) && c[l] < least) {
            best = l;
            least = c[l];
          }
        if (best < 0) {
          if (c[0] < kNever || c[kSmallLevel] < kNever) return kNever;
          continue;  // no pairs
        }
        sum += least;
        needI[a] |= 1u << best;
        (k.self ? needI : needJ)[b] |= 1u << best;
        if (write) {
          k.level[a][b] = best;
          k.cands += found[at(best, a, b)];
        }
      }
    for (int q = 0; q < (k.self || J.prepared ? 1 : 2); ++q)
      for (int c = 0; c < kClasses; ++c) {
        const double n = (double)(cr[q].row[c + 1] - cr[q].row[c]);
        const double len = q == 0 ? I.len[c] : J.len[c];
        for (int l = 0; l < kFoldLevels; ++l)
          if (((q == 0 ? needI : needJ)[c] >> l) & 1u)
            sum += n * (kFoldEntryNs * len + kFoldColumnNs * fold_k(MIXED, l));
      }
    return sum;
  };
  // levels whose tiles save less than folding the rows for them costs go
  uint32_t use = all;
  double total = choose(use, false);
  for (int l = 0; l < kFoldLevels; ++l) {
    const uint32_t fewer = use & ~(1u << l);
    if (fewer == use || fewer == 0) continue;
    const double c = choose(fewer, false);
    if (c < total) {
      total = c;
      use = fewer;
    }
  }
  k.cost = choose(use, true);
  return CUAPSS_OK;
}

int class_of(const FoldSide& s, int block) {
  int c = 0;
  while (c + 1 < kClasses && block >= s.edge[c + 1]) ++c;
  return c;
}

// Allocates and builds the folded levels a side needs, per class.
template <bool MIXED>
cuapss_status build_levels(FoldSide& s, const uint32_t (&need)[kClasses], const int32_t* perm,
                           const FoldAlloc& alloc, Workspace& ws, const std::string& tag,
                           cudaStream_t st) {
  // one allocation for all levels: which levels a call takes varies from input
  // to input more than their total does
  size_t size[kFoldLevels] = {}, total = 0;
  for (int l = 0; l < kFoldLevels; ++l) {
    int lo = s.nb, hi = 0;
    for (int c = 0; c < kClasses; ++c)
      if (s.edge[c + 1] > s.edge[c] && ((need[c] >> l) & 1u)) {
        lo = std::min(lo, s.edge[c]);
        hi = std::max(hi, s.edge[c + 1]);
      }
    if (hi <= lo) continue;
    s.out.first[l] = lo;
    size[l] = (size_t)(hi - lo) * fold_bytes(MIXED, l);
    total += size[l];
  }
  void* p = nullptr;
  ST_TRY(alloc("levels", total, &p));
  uint8_t* at = static_cast<uint8_t*>(p);
  for (int l = 0; l < kFoldLevels; ++l) {
    s.out.base[l] = size[l] ? at : nullptr;
    at += size[l];
  }
  std::vector<uint16_t> masks((size_t)s.nb, 0);
  for (int c = 0; c < kClasses; ++c)
    for (int b = s.edge[c]; b < s.edge[c + 1]; ++b) masks[(size_t)b] = (uint16_t)need[c];
  return fold_places<MIXED>(s, s.rowmap, (int64_t)s.nb * kBlockRows, masks, 0, perm, s.out, ws,
                            tag, st);
}

// Units: windows of J blocks from the long rows down (the costly units
// first), in each window every I pair against each class's part of it, so
// that the CTAs running at one time share a window's chunks in L2. Wider
// folds get proportionally shorter ranges.
template <bool MIXED>
void make_units(FoldTask& k, int sms) {
  const FoldSide& I = *k.I;
  const FoldSide& J = *k.J;
  const int nbJ = J.nb;
  const int pair = kPair<MIXED>;
  const double total = k.self ? 0.5 * nbJ * (nbJ + 2.0) / pair : std::ceil((double)I.nb / pair) * nbJ;
  const int w = (int)std::max(1.0, std::min(MIXED ? 128.0 : 32.0, total / (sms * 16.0)));
  for (int j1 = nbJ; j1 > 0; j1 -= w) {
    const int j0 = std::max(0, j1 - w);
    for (int b = class_of(J, j1 - 1); b >= 0 && J.edge[b + 1] > j0; --b) {
      const int s0 = std::max(j0, J.edge[b]), s1 = std::min(j1, J.edge[b + 1]);
      if (s0 >= s1) continue;
      int a = 0;
      for (int i = 0; i < (k.self ? std::min(I.nb, s1) : I.nb); i += pair) {
        while (i >= I.edge[a + 1]) ++a;
        const int lv = k.level[a][b];
        const int f0 = k.self ? std::max(s0, i) : s0;
        // the pair's second block reaches at least as far
        const int e1 = k.last.empty() ? s1
                                      : std::min(s1, k.last[(size_t)std::min(I.nb, i + pair) - 1] + 1);
        const double rel = tile_cost<MIXED>(lv) / tile_cost<MIXED>(MIXED ? 1 : 3);
        const int step = std::max(1, (int)(w / std::max(1.0, rel)));
        for (int f = f0; f < e1; f += step) {
          const int len = std::min(e1 - f, step);
          // spread the starts of neighbouring units over the range
          const int turn = (int)(((int64_t)(k.units.size() % 16) * len) / 16);
          k.units.push_back(make_int4(i, f, f + len, lv | turn << 8));
        }
      }
    }
  }
  k.tiles = k.self ? (int64_t)nbJ * (nbJ + 1) / 2 : (int64_t)I.nb * nbJ;
}

// Widths for sides too small to sample: one for all.
void one_level(FoldTask& k) {
  for (auto& row : k.level)
    for (int& l : row) l = kSmallLevel;  // K = 256 or 64
}

// The candidates, among so many pairs of rows of mean length len, at which an
// unsampled join stops being faster than the probing path by gain_ns. 0: it is
// not worth a try, three times as many are expected (2,000 rows of 800 entries
// at t = 0.5, mixed: 2.0 ms probing, 9.0 folded with every pair a candidate).
int64_t small_limit(cuapss_ctx* ctx, double len, double pairs, double expected, double gain_ns) {
  double n = 0.0;
  for (int it = 0; it < 4; ++it) {
    n = std::min((double)kSmallMaxCand,
                 gain_ns * ctx->sms / cand_ns(len, n / std::max(pairs, 1.0)));
  }
  return expected > 3.0 * n ? 0 : (int64_t)n;
}

// The levels the sides of a task need, per class.
void needed(const FoldTask& k, uint32_t (&needI)[kClasses], uint32_t (&needJ)[kClasses]) {
  for (int x = 0; x < kClasses; ++x)
    for (int y = k.self ? x : 0; y < kClasses; ++y) {
      if (k.I->edge[x + 1] <= k.I->edge[x] || k.J->edge[y + 1] <= k.J->edge[y]) continue;
      needI[x] |= 1u << k.level[x][y];
      needJ[y] |= 1u << k.level[x][y];
    }
  if (k.self)
    for (int c = 0; c < kClasses; ++c) needI[c] |= needJ[c];
}

cuapss_status upload_units(std::vector<FoldTask>& tasks, Workspace& ws, cudaStream_t st) {
  std::vector<int4> all;
  for (FoldTask& k : tasks) all.insert(all.end(), k.units.begin(), k.units.end());
  int4* d = nullptr;
  ST_TRY(ws.get("tiles:units", std::max<size_t>(all.size(), 1), &d));
  if (!all.empty())
    CU_TRY(cudaMemcpyAsync(d, all.data(), sizeof(int4) * all.size(), cudaMemcpyHostToDevice, st));
  for (FoldTask& k : tasks) {
    k.d_units = d;
    d += k.units.size();
  }
  return CUAPSS_OK;
}

// Candidate lists above this ask for the free memory first and take at most
// this share of it.
constexpr double kAskBytes = 1e9, kListShare = 0.6;

// Tiles and verification of all tasks into one unsorted pair list. *done =
// false: the candidates do not fit what a folded join may take.
template <bool MIXED>
cuapss_status run_tasks(cuapss_ctx* ctx, std::vector<FoldTask>& tasks, double nrm2,
                        const VerifyArgs& common, int64_t max_cand, FoldResult* r, bool* done) {
  *done = false;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const size_t nt = tasks.size();
  // control words: pairs found, then per task candidates, {unit counter,
  // verify's group counter}, error flags
  unsigned long long* ctl = nullptr;
  ST_TRY(ws.get("fold:ctl", 1 + 3 * nt, &ctl));
  std::vector<unsigned long long> h(1 + 3 * nt);
  // sizes in steps of a quarter of their power of two, so that calls of similar
  // inputs find their buffers large enough; room that earlier calls left is
  // room to use (as it is: no call asks for more because of it), but the route
  // is decided by the caps that a new context would have
  for (FoldTask& k : tasks) {
    int64_t step = 1 << 16;
    while (step * 8 <= k.cap) step *= 2;
    k.cap = (k.cap + step - 1) / step * step;
  }
  std::vector<int64_t> own;
  for (const FoldTask& k : tasks) own.push_back(k.cap);
  if (nt == 1)
    tasks[0].cap = std::max<int64_t>(
        tasks[0].cap, (int64_t)std::min({ws.held("fold:cand") / 8, ws.held("out:key") / 8,
                                         ws.held("out:idx") / 4, ws.held("out:sim") / 4}));
  for (int attempt = 0; attempt < 3; ++attempt) {
    int64_t most = 1, room = 0;
    for (FoldTask& k : tasks) {
      most = std::max(most, k.cap);
      room += k.cap;
    }
    if (room >= (int64_t)UINT32_MAX) return CUAPSS_OK;  // out_idx
    // large lists leave the sorted result its room (at most 24 bytes a pair,
    // of which there are half as many as the first list's slots)
    const double bytes = 8.0 * (double)most + 16.0 * (double)room;
    if (bytes > kAskBytes) {
      size_t free_b = 0, total_b = 0;
      CU_TRY(cudaMemGetInfo(&free_b, &total_b));
      const double held = (double)(ws.held("fold:cand") + ws.bytes_held("out:"));
      if (bytes > kListShare * ((double)free_b + held)) return CUAPSS_OK;
    }
    uint64_t* cand = nullptr;
    ST_TRY(ws.get("fold:cand", (size_t)most, &cand));  // the tasks run one after another
    ST_TRY(ws.get("out:key", (size_t)room, &r->okey));
    ST_TRY(ws.get("out:idx", (size_t)room, &r->oidx));
    ST_TRY(ws.get("out:sim", (size_t)room, &r->osim));
    CU_TRY(cudaMemsetAsync(ctl, 0, 8 * (1 + 3 * nt), st));
    for (size_t i = 0; i < nt; ++i) {
      FoldTask& k = tasks[i];
      FoldTileArgs ta;
      for (int l = 0; l < kFoldLevels; ++l) {
        FoldLevel& L = ta.lev[l];
        L.I = k.I->out.base[l];
        L.J = k.J->out.base[l];
        L.firstI = k.I->out.first[l];
        L.firstJ = k.J->out.first[l];
        L.nkc = fold_k(MIXED, l) / kChunk<MIXED>;
        L.eps = fold_eps(MIXED, l, nrm2, k.t_min, k.I->x.nonneg, k.J->x.nonneg);
        if (L.I) r->max_band = std::max(r->max_band, (double)L.eps);
      }
      ta.nI = k.I->slots ? k.I->slots : k.I->x.n;
      ta.nJ = k.J->slots ? k.J->slots : k.J->x.n;
      ta.nbI = k.I->nb;
      ta.nbJ = k.J->nb;
      ta.self = k.self ? 1 : 0;
      ta.t = k.t;
      ta.t_row = k.J->t_place;
      ta.units = k.d_units;
      ta.nunits = (int)k.units.size();
      ta.cand = cand;
      ta.cand_cap = k.limit > 0 ? k.limit : k.cap;
      // (what makes a sampled batch probe, below; for the other joins, whose
      // samples see all their rows, the look at the count costs 8 of the 480 us
      // of a 256-row index query)
      ta.give_up_at = k.limit > 0 ? k.limit : k.J->t_place ? std::max(max_cand, own[i]) : 0;
      ta.cand_count = ctl + 1 + 3 * i;
      ta.unit_counter = reinterpret_cast<int*>(ctl + 2 + 3 * i);
      ta.err = reinterpret_cast<int*>(ctl + 3 + 3 * i);
      ST_TRY(launch_fold<MIXED>(ta, ctx->sms, st, false));
      VerifyArgs va = common;
      va.cand = cand;
      va.ncand = ctl + 1 + 3 * i;
      va.cap = ta.cand_cap;
      va.work = reinterpret_cast<unsigned*>(ctl + 2 + 3 * i) + 1;
      va.permI = k.I->rowmap;
      va.permJ = k.J->rowmap;
      va.rpI = k.I->x.rp;
      va.colI = k.I->x.col;
      va.valI = k.I->x.val;
      va.rpJ = k.J->x.rp;
      va.colJ = k.J->x.col;
      va.valJ = k.J->x.val;
      va.self = ta.self;
      va.j_offset = k.j_offset;
      va.out_key = r->okey;
      va.out_idx = r->oidx;
      va.out_sim = r->osim;
      va.out_count = ctl;
      ST_TRY(launch_verify(va, st));
    }
    // (while the kernels run: counted as the units were made it took 5 of the
    // 370 us of a 20,000-row join)
    if (attempt == 0)
      for (const FoldTask& k : tasks) k.count_tiles(kPair<MIXED>, r->level_tiles);
    CU_TRY(cudaMemcpyAsync(h.data(), ctl, 8 * (1 + 3 * nt), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    bool over = false, past_own = false, given_up = false;
    int64_t want = 0;
    for (size_t i = 0; i < nt; ++i) {
      const int herr = (int)h[3 + 3 * i];
      if (herr & kErrTimeout) return CUAPSS_ETIMEOUT;
      if (herr) return CUAPSS_ECUDA;
      const int64_t c = (int64_t)h[1 + 3 * i];
      want += c;
      over = over || c > tasks[i].cap;
      past_own = past_own || c > own[i];
      given_up = given_up || (tasks[i].limit > 0 && c > tasks[i].limit);
      tasks[i].cap = std::max(tasks[i].cap, c);
    }
    r->npairs = (int64_t)h[0];
    r->ncand = want;
    if (given_up || (past_own && want > max_cand)) return CUAPSS_OK;
    if (!over) {
      *done = true;
      return CUAPSS_OK;
    }
  }
  return CUAPSS_OK;
}

// FoldTask::last of a self-join whose rows are sorted by length.
cuapss_status block_reach(cuapss_ctx* ctx, FoldTask& k, double nrm2) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  FoldSide& I = *k.I;
  const int nb = I.nb;
  // T = (t / norm)^2 with room for the rounding of t, of the norm and of the
  // reported sums, in the fixed point of the squares
  const double T = ((double)k.t - 1e-6) * ((double)k.t - 1e-6) / nrm2 * (1.0 - 1e-5);
  if (!(T > 0.0) || T >= 1.9) return CUAPSS_OK;
  int* d = nullptr;
  ST_TRY(ws.get("fold:need", 2 * (size_t)nb, &d));
  CU_TRY(cudaMemsetAsync(d, 0x3f, 4 * (size_t)nb, st));
  CU_TRY(cudaMemsetAsync(d + nb, 0, 4 * (size_t)nb, st));
  const int64_t slots = (int64_t)nb * kBlockRows;
  k_block_needs<<<grid_for(slots * 32, kThreads), kThreads, 0, st>>>(
      I.rowmap, slots, I.x.rp, I.x.val, (uint32_t)(T * kSquareScale), d, d + nb);
  LAUNCH_CHECK();
  std::vector<int> h(2 * (size_t)nb);
  CU_TRY(cudaMemcpyAsync(h.data(), d, 8 * (size_t)nb, cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  // first[J]: the first I block with a row long enough for some row of J or of
  // a later block
  std::vector<int> first((size_t)nb);
  int i = 0, longest = h[(size_t)nb];
  std::vector<int> need(h.begin(), h.begin() + nb);
  for (int j = nb - 2; j >= 0; --j) need[(size_t)j] = std::min(need[(size_t)j], need[(size_t)j + 1]);
  for (int j = 0; j < nb; ++j) {
    while (i < j && longest < need[(size_t)j]) longest = std::max(longest, h[(size_t)nb + ++i]);
    first[(size_t)j] = i;
  }
  // first is non-decreasing: the last J of each I
  k.last.assign((size_t)nb, nb - 1);
  for (int q = 0, j = 0; q < nb; ++q) {
    j = std::max(j, q);
    while (j + 1 < nb && first[(size_t)j + 1] <= q) ++j;
    k.last[(size_t)q] = j;
  }
  return CUAPSS_OK;
}

template <bool MIXED>
cuapss_status join_fold_as(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                           const int32_t* perm, double nrm2, const CostFn& other_ns, FoldResult* r,
                           bool* done) {
  *done = false;
  const bool self = b == nullptr;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  FoldSide SI, SJ;
  SI.x = a;
  if (!self) SJ.x = *b;
  std::vector<FoldTask> tasks(1);
  FoldTask& k = tasks[0];
  k.I = &SI;
  k.J = self ? &SI : &SJ;
  k.self = self;
  k.t = t;
  const int64_t nbI = ceil_div(SI.x.n, kBlockRows), nbJ = ceil_div(k.J->x.n, kBlockRows);
  const double tiles128 = self ? 0.5 * nbI * (nbI + 1.0) : (double)nbI * nbJ;
  const bool sampled = tiles128 >= kSampleMinTiles;
  auto allocI = [&ws](const std::string& name, size_t bytes, void** out) {
    return ws.get("fold:I:" + name, bytes, out);
  };
  auto allocJ = [&ws](const std::string& name, size_t bytes, void** out) {
    return ws.get("fold:J:" + name, bytes, out);
  };
  const double probing_gain =
      kProbeFixedNs + kProbeEntryNs * (double)(a.nnz + (self ? 0 : b->nnz));
  if (!sampled) {
    const double n = (double)a.n, pairs = self ? 0.5 * n * (n - 1.0) : n * (double)b->n;
    const double len = self ? mean_len(a) : 0.5 * (mean_len(a) + mean_len(*b));
    k.limit = small_limit(ctx, len, pairs, pairs * passing_share(len, fold_k(MIXED, kSmallLevel), t),
                          probing_gain);
    if (k.limit == 0) return CUAPSS_OK;
  }
  ST_TRY(order_side(SI, sampled, allocI, ws, "fold:I", st));
  if (!self) ST_TRY(order_side(SJ, sampled, allocJ, ws, "fold:J", st));
  if (sampled) {
    ST_TRY(plan_levels<MIXED>(ctx, k, perm, nrm2));
    double ns = 0.0;
    ST_TRY(other_ns(&ns));
    if (k.cost >= tiles128 * ns + probing_gain * ctx->sms) return CUAPSS_OK;
  } else {
    one_level(k);
  }
  // (a launch and a round trip: 60 us)
  if (self && sampled && k.cost > kReachMinNs * ctx->sms) ST_TRY(block_reach(ctx, k, nrm2));
  uint32_t needI[kClasses] = {}, needJ[kClasses] = {};
  needed(k, needI, needJ);
  ST_TRY(build_levels<MIXED>(SI, needI, perm, allocI, ws, "fold:I", st));
  if (!self) ST_TRY(build_levels<MIXED>(SJ, needJ, perm, allocJ, ws, "fold:J", st));
  make_units<MIXED>(k, ctx->sms);
  ST_TRY(upload_units(tasks, ws, st));
  r->tiles = k.tiles;
  r->rbitsI = std::max(1, bits_for((uint64_t)SI.x.n));
  r->rbitsJ = std::max(1, bits_for((uint64_t)k.J->x.n));
  // twice what the sample promises: a run that does not fit is run again
  const int64_t expect = std::max<int64_t>((int64_t)(2.0 * k.cands), 1 << 20);
  k.cap = sampled ? expect + SI.x.n + k.J->x.n : k.limit;
  VerifyArgs va;
  va.t = t;
  va.rbits = r->rbitsJ;
  // a join whose sample misjudged it is left to the probing path
  return run_tasks<MIXED>(ctx, tasks, nrm2, va, 4 * expect, r, done);
}

// ---- resident index -------------------------------------------------------
// Levels a segment holds for its classes: narrow ones for every row, wide
// ones for the long rows.
template <bool MIXED>
uint32_t index_levels(int c, bool sampled) {
  if (!sampled) return 1u << kSmallLevel;
  // mixed: 64, 128, 256 | 512 | 1,024 | 2,048; FP32: 32, 64, 128 | 256 | 512 | 1,024
  const uint32_t base = MIXED ? 0x0bu : 0x2au;
  const uint32_t wide[3] = {MIXED ? 1u << 6 : 1u << 7, 1u << 8, 1u << 9};
  return base | (c >= 6 ? wide[0] : 0) | (c >= 9 ? wide[1] : 0) | (c >= 13 ? wide[2] : 0);
}

template <bool MIXED>
cuapss_status fold_index_as(cuapss_ctx* ctx, const DevCsr& x, const int32_t* perm,
                            const FoldAlloc& alloc, FoldSide* s) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  s->x = x;
  s->prepared = true;
  const bool sampled = ceil_div(x.n, kBlockRows) >= 2 * kClasses;
  ST_TRY(order_side(*s, sampled, alloc, ws, "fold:X", st));
  uint32_t need[kClasses];
  uint32_t all = 0;
  for (int c = 0; c < kClasses; ++c) {
    need[c] = s->levels[c] = index_levels<MIXED>(c, sampled);
    all |= need[c];
  }
  ST_TRY(build_levels<MIXED>(*s, need, perm, alloc, ws, "fold:X", st));
  if (!sampled) return CUAPSS_OK;
  unsigned long long* len_sum = nullptr;
  ST_TRY(ws.get("fold:xlen", kClasses, &len_sum));
  CU_TRY(cudaMemsetAsync(len_sum, 0, 8 * kClasses, st));
  ST_TRY(sample_side<MIXED>(*s, all, len_sum, perm, alloc, ws, "fold:X", st));
  unsigned long long h[kClasses];
  CU_TRY(cudaMemcpyAsync(h, len_sum, sizeof(h), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  const ClassRows cr = class_rows(*s);
  for (int c = 0; c < kClasses; ++c) {
    const int64_t m = std::min<int64_t>(kBlockRows, cr.row[c + 1] - cr.row[c]);
    s->len[c] = m > 0 ? (double)h[c] / (double)m : 0.0;
  }
  return CUAPSS_OK;
}

template <bool MIXED>
cuapss_status fold_query_as(cuapss_ctx* ctx, const std::vector<FoldSegment>& segs,
                            const DevCsr& q, const float* t, const float* t_row,
                            const int32_t* perm, double nrm2, double other_ns, int64_t rows,
                            FoldResult* r, bool* done) {
  *done = false;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  FoldSide Q;
  Q.x = q;
  Q.t_row = t_row;
  auto alloc = [&ws](const std::string& name, size_t bytes, void** out) {
    return ws.get("fold:Q:" + name, bytes, out);
  };
  // several blocks of queries: those with much to compare together
  ST_TRY(order_side(Q, q.n > 2 * kBlockRows, alloc, ws, "fold:Q", st));
  const float t_min = *std::min_element(t, t + q.n);
  std::vector<FoldTask> tasks(segs.size());
  // unsampled segments: their candidates together have one limit
  auto is_sampled = [&](const FoldSide& s) {
    return s.sample != nullptr && (double)Q.nb * s.nb >= kSampleMinTiles;
  };
  double small_rows = 0.0, small_nnz = 0.0;
  for (const FoldSegment& g : segs)
    if (!is_sampled(*g.side)) {
      small_rows += (double)g.side->x.n;
      small_nnz += (double)g.side->x.nnz;
    }
  int64_t limit = 0;
  if (small_rows > 0) {
    const double len = 0.5 * (mean_len(q) + small_nnz / small_rows);
    double expected = 0.0;
    for (int64_t i = 0; i < q.n; ++i)
      expected += small_rows * passing_share(len, fold_k(MIXED, kSmallLevel), t[i]);
    limit = small_limit(ctx, len, small_rows * (double)q.n, expected, kProbeFixedNs);
    if (limit == 0) return CUAPSS_OK;
  }
  uint32_t needQ[kClasses] = {};
  double cost = 0.0;
  int64_t max_cand = kSmallMaxCand;
  r->tiles = 0;
  for (size_t i = 0; i < segs.size(); ++i) {
    FoldTask& k = tasks[i];
    k.I = &Q;
    k.J = segs[i].side;
    k.t = 1.0f;
    k.t_min = t_min;
    k.j_offset = segs[i].row0;
    const double tiles128 = (double)Q.nb * k.J->nb;
    if (is_sampled(*k.J)) {
      ST_TRY(plan_levels<MIXED>(ctx, k, perm, nrm2));
      cost += k.cost;
    } else {
      one_level(k);
      cost += tiles128 * tile_cost<MIXED>(kSmallLevel) / kPair<MIXED>;
      k.limit = std::max<int64_t>(1, (int64_t)((double)limit * (double)k.J->x.n / small_rows));
    }
    uint32_t needJ[kClasses] = {};
    needed(k, needQ, needJ);
    make_units<MIXED>(k, ctx->sms);
    r->tiles += k.tiles;
    k.cap = k.limit > 0 ? k.limit : std::max<int64_t>((int64_t)(2.0 * k.cands), 1 << 18);
    max_cand = std::max(max_cand, 4 * k.cap);
  }
  if (cost >= (double)r->tiles * other_ns + kProbeFixedNs * ctx->sms) return CUAPSS_OK;
  ST_TRY(build_levels<MIXED>(Q, needQ, perm, alloc, ws, "fold:Q", st));
  ST_TRY(upload_units(tasks, ws, st));
  r->rbitsI = std::max(1, bits_for((uint64_t)q.n));
  r->rbitsJ = std::max(1, bits_for((uint64_t)std::max<int64_t>(rows, 1)));
  VerifyArgs va;
  va.t_of_i = t_row;
  va.rbits = r->rbitsJ;
  return run_tasks<MIXED>(ctx, tasks, nrm2, va, max_cand, r, done);
}

// ---- batches ---------------------------------------------------------------
// The batch's pairs in order of their threshold make kBatchT classes of equal
// size. Up to kBatchRows rows of the instance in the middle of each class are
// compared with one another at the class's lowest threshold: rows of different
// instances never meet, and their products say nothing about those that do
// (instances of 10 and of 300 entries a row in one batch).
constexpr int kBatchT = kClasses;
constexpr int kBatchRows = 2 * kBlockRows;
constexpr int kBatchBlocks = kBatchT * kBatchRows / kBlockRows;
constexpr double kSmallBatchNs = 1e6;

template <bool MIXED>
cuapss_status fold_batch_as(cuapss_ctx* ctx, const DevCsr& x, int k, const int64_t* inst_ptr,
                            const float* t, const int32_t* perm, double nrm2, double other_ns,
                            std::vector<int>* width, FoldResult* r, bool* done) {
  *done = false;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const int pair = kPair<MIXED>;
  // ---- instances with pairs, by threshold
  std::vector<int> inst;
  double all_pairs = 0.0;
  for (int q = 0; q < k; ++q) {
    const double n = (double)(inst_ptr[q + 1] - inst_ptr[q]);
    if (n < 2) continue;
    inst.push_back(q);
    all_pairs += n * n;
  }
  width->assign((size_t)k, 0);
  if (inst.empty()) return CUAPSS_OK;
  std::sort(inst.begin(), inst.end(), [&](int a, int b) { return t[a] != t[b] ? t[a] < t[b] : a < b; });
  float grid[kBatchT];  // each class's lowest threshold
  int mid[kBatchT];     // and its sampled instance
  {
    double seen = 0.0;
    int g = 0, m = 0;
    for (int q : inst) {
      const double n = (double)(inst_ptr[q + 1] - inst_ptr[q]);
      while (g < kBatchT && seen >= all_pairs * g / kBatchT) grid[g++] = t[q];
      seen += n * n;
      while (m < kBatchT && seen > all_pairs * (m + 0.5) / kBatchT) mid[m++] = q;
    }
    while (g < kBatchT) grid[g++] = t[inst.back()];
    while (m < kBatchT) mid[m++] = inst.back();
  }
  // ---- shares of their pairs at or above those thresholds, per level
  double tiles = 0.0;
  for (int q : inst) {
    const double nb = (double)ceil_div(inst_ptr[q + 1] - inst_ptr[q], kBlockRows);
    tiles += 0.5 * nb * (nb + 1.0);
  }
  // what probing would take; a sampled tile gets no more than a tenth of it
  const double probing_ns =
      tiles * other_ns / ctx->sms + kProbeFixedNs + kBatchProbeEntryNs * (double)x.nnz;
  // (below kSmallBatchNs only those that the mean length calls for: 14 instances
  // of 64 .. 2,702 rows of 30 entries: 248 us, 286 with all of them sampled)
  uint32_t all = sampled_levels<MIXED>(0.1 * probing_ns);
  if (MIXED && probing_ns < kSmallBatchNs)
    all &= ((2u << kSmallLevel) - 1u) |
           useful_levels<MIXED>(mean_len(x), t[inst.front()], 0.5 * all_pairs, ctx->sms);
  const int64_t slots = (int64_t)kBatchBlocks * kBlockRows;
  std::vector<int32_t> rows((size_t)slots, -1);
  std::vector<float> ht((size_t)slots);
  for (int g = 0; g < kBatchT; ++g) {
    const int64_t first = inst_ptr[mid[g]], n = inst_ptr[mid[g] + 1] - first;
    for (int64_t i = 0; i < kBatchRows; ++i) {
      // evenly spaced; classes that share an instance take different rows
      const int64_t r = n >= kBatchRows ? ((i * kBatchT + g) * n) / (kBatchRows * kBatchT) : i;
      if (r < n) rows[(size_t)(g * kBatchRows + i)] = (int32_t)(first + r);
      ht[(size_t)(g * kBatchRows + i)] = grid[g];
    }
  }
  const size_t ncnt = (size_t)kFoldLevels * kBatchBlocks * kBatchBlocks;
  unsigned long long* stats = nullptr;  // control words, counts
  ST_TRY(ws.get("fold:stats", 1 + ncnt / 2, &stats));
  CU_TRY(cudaMemsetAsync(stats, 0, 8 + 4 * ncnt, st));
  FoldSide B;
  B.x = x;
  int32_t* sample = nullptr;
  float* sample_t = nullptr;
  ST_TRY(ws.get("fold:sI:sample", (size_t)slots, &sample));
  ST_TRY(ws.get("fold:sI:t", (size_t)slots, &sample_t));
  CU_TRY(cudaMemcpyAsync(sample, rows.data(), 4 * (size_t)slots, cudaMemcpyHostToDevice, st));
  CU_TRY(cudaMemcpyAsync(sample_t, ht.data(), 4 * (size_t)slots, cudaMemcpyHostToDevice, st));
  FoldOut so;
  uint8_t* samples = nullptr;
  ST_TRY(ws.get("fold:sI:samples", kBatchBlocks * fold_offset_bytes(MIXED, kFoldLevels), &samples));
  for (int l = 0; l < kFoldLevels; ++l)
    so.base[l] = samples + kBatchBlocks * fold_offset_bytes(MIXED, l);
  ST_TRY(fold_places<MIXED>(B, sample, slots, {}, all, perm, so, ws, "fold:sI", st));
  FoldTileArgs ta;
  std::vector<int4> units;
  for (int l = kFoldLevels - 1; l >= 0; --l) {
    if (!((all >> l) & 1u)) continue;
    ta.lev[l].I = ta.lev[l].J = so.base[l];
    ta.lev[l].nkc = fold_k(MIXED, l) / kChunk<MIXED>;
    ta.lev[l].eps = fold_eps(MIXED, l, nrm2, 1.0, x.nonneg, x.nonneg);
    for (int a = 0; a < kBatchBlocks; a += pair)
      for (int b = a; b < a / 2 * 2 + 2; ++b) units.push_back(make_int4(a, b, b + 1, l));
  }
  int4* d_units = nullptr;
  ST_TRY(ws.get("fold:sunits", units.size(), &d_units));
  CU_TRY(cudaMemcpyAsync(d_units, units.data(), sizeof(int4) * units.size(),
                         cudaMemcpyHostToDevice, st));
  ta.nI = ta.nJ = slots;
  ta.nbI = ta.nbJ = kBatchBlocks;
  ta.self = 1;
  ta.t_row = sample_t;
  ta.units = d_units;
  ta.nunits = (int)units.size();
  ta.unit_counter = reinterpret_cast<int*>(stats);
  ta.err = ta.unit_counter + 1;
  ta.class_count = reinterpret_cast<uint32_t*>(stats + 1);
  ST_TRY(launch_fold<MIXED>(ta, ctx->sms, st, true));
  static_assert(8 + 4 * kFoldLevels * kBatchBlocks * kBatchBlocks <= kPinnedBytes, "pinned scratch");
  const auto* h = static_cast<const unsigned long long*>(ctx->pinned);
  CU_TRY(cudaMemcpyAsync(ctx->pinned, stats, 8 + 4 * ncnt, cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  const int herr = (int)(h[0] >> 32);
  if (herr & kErrTimeout) return CUAPSS_ETIMEOUT;
  if (herr) return CUAPSS_ECUDA;
  const uint32_t* hc = reinterpret_cast<const uint32_t*>(h + 1);
  const double mean = mean_len(x);
  double share[kFoldLevels][kBatchT];
  for (int l = 0; l < kFoldLevels; ++l)
    for (int g = 0; g < kBatchT; ++g) {
      const double m = (double)std::min<int64_t>(kBatchRows, inst_ptr[mid[g] + 1] - inst_ptr[mid[g]]);
      double c = 0.0;
      for (int a = 2 * g; a < 2 * g + 2; ++a)
        for (int b = a; b < 2 * g + 2; ++b)
          c += (double)hc[((size_t)l * kBatchBlocks + a) * kBatchBlocks + b];
      share[l][g] = std::max(c, 0.5) / (0.5 * m * (m - 1.0));
    }
  // ---- a level per instance; instances laid out level by level
  std::vector<int> lev((size_t)k, 0);
  double cost = 0.0, cands = 0.0;
  std::vector<int> by_level[kFoldLevels];
  int g = 0;
  for (int q : inst) {
    while (g + 1 < kBatchT && grid[g + 1] <= t[q]) ++g;
    // the classes of the instance's threshold and their neighbours: several
    // instances' shares
    int g0 = g;
    while (g0 > 0 && grid[g0 - 1] == grid[g]) --g0;
    g0 = std::max(0, g0 - 1);
    const int g1 = std::min(kBatchT - 1, g + 1);
    const int64_t n = inst_ptr[q + 1] - inst_ptr[q];
    const double nb = (double)ceil_div(n, kBlockRows);
    const double pairs = 0.5 * (double)n * (double)(n - 1);
    double best = 1e300, best_cand = 0.0;
    for (int l = 0; l < kFoldLevels; ++l) {
      if (!((all >> l) & 1u)) continue;
      double sum = 0.0;
      for (int c = g0; c <= g1; ++c) sum += share[l][c];
      const double passing = sum / (g1 - g0 + 1), cand = passing * pairs;
      const double ns = std::ceil(nb / pair) * (nb + 1.0) * 0.5 * tile_cost<MIXED>(l) +
                        cand * cand_ns(mean, passing) +
                        (double)n * (mean * kFoldEntryNs + fold_k(MIXED, l) * kFoldColumnNs);
      if (ns < best) {
        best = ns;
        best_cand = cand;
        lev[(size_t)q] = l;
      }
    }
    cost += best;
    cands += best_cand;
    by_level[lev[(size_t)q]].push_back(q);
  }
  if (cost >= probing_ns * ctx->sms) return CUAPSS_OK;
  std::vector<int64_t> tab;
  std::vector<FoldTask> tasks(1);
  FoldTask& task = tasks[0];
  task.I = task.J = &B;
  task.self = true;
  int64_t S = 0;
  size_t size[kFoldLevels] = {}, total = 0;
  std::vector<uint16_t> masks;
  const int most = (int)std::max(1.0, std::min(64.0, tiles / pair / (ctx->sms * 16.0)));
  for (int l = kFoldLevels - 1; l >= 0; --l) {  // the costly ones first
    B.out.first[l] = (int)(S / kBlockRows);
    for (int q : by_level[l]) {
      const int64_t n = inst_ptr[q + 1] - inst_ptr[q];
      int tbits = 0;
      memcpy(&tbits, &t[q], sizeof(float));
      tab.insert(tab.end(), {S, inst_ptr[q], n, (int64_t)tbits});
      const int b0 = (int)(S / kBlockRows), b1 = b0 + (int)ceil_div(n, kBlockRows);
      for (int i = b0; i < b1; i += pair) {
        const int single = MIXED && i + 1 >= b1 ? kFoldSingle : 0;
        for (int f = i; f < b1; f += most)
          task.units.push_back(make_int4(i, f, std::min(b1, f + most), l | single));
      }
      task.tiles += (int64_t)(b1 - b0) * (b1 - b0 + 1) / 2;
      (*width)[(size_t)q] = fold_k(MIXED, l);
      masks.insert(masks.end(), (size_t)(b1 - b0), (uint16_t)(1u << l));
      S += (int64_t)(b1 - b0) * kBlockRows;
      if (S >= INT32_MAX) return CUAPSS_OK;  // the probing path takes a bucket at a time
    }
    size[l] = (size_t)(S / kBlockRows - B.out.first[l]) * fold_bytes(MIXED, l);
    total += size[l];
  }
  uint8_t* levels = nullptr;
  ST_TRY(ws.get("fold:B:levels", total, &levels));
  for (int l = 0; l < kFoldLevels; ++l) {
    if (size[l]) B.out.base[l] = levels;
    levels += size[l];
  }
  B.nb = (int)(S / kBlockRows);
  B.slots = S;
  const int kq = (int)inst.size();
  int64_t* d_tab = nullptr;
  float* t_place = nullptr;
  ST_TRY(ws.get("fold:B:tab", tab.size(), &d_tab));
  ST_TRY(ws.get("fold:B:map", (size_t)S, &B.rowmap));
  ST_TRY(ws.get("fold:B:t", (size_t)S, &t_place));
  CU_TRY(cudaMemcpyAsync(d_tab, tab.data(), 8 * tab.size(), cudaMemcpyHostToDevice, st));
  k_batch_places<<<grid_for((int64_t)kq, 1), kThreads, 0, st>>>(d_tab, kq, B.rowmap, t_place);
  LAUNCH_CHECK();
  B.t_place = t_place;
  ST_TRY(fold_places<MIXED>(B, B.rowmap, S, masks, 0, perm, B.out, ws, "fold:B", st));
  const int64_t expect = std::max<int64_t>((int64_t)(2.0 * cands), 1 << 20);
  task.cap = expect + x.n;
  ST_TRY(upload_units(tasks, ws, st));
  r->tiles = task.tiles;
  r->rbitsI = r->rbitsJ = std::max(1, bits_for((uint64_t)x.n));
  VerifyArgs va;
  va.t_row = t_place;
  va.rbits = r->rbitsJ;
  return run_tasks<MIXED>(ctx, tasks, nrm2, va, 4 * expect, r, done);
}

// Verification holds a row's first entry in 32 bits; a longer matrix is left
// to the probing path, which compacts it (batches) or refuses it.
bool verifiable(const DevCsr& x) { return x.nnz < (int64_t)UINT32_MAX; }

// Folded joins take more working memory than probing ones where the bound
// prunes less (24 bytes a candidate). One that does not get it frees what it
// took and leaves the call to the probing path, during which its buffers may
// go.
class FoldMemory {
 public:
  explicit FoldMemory(Workspace& ws) : ws_(ws) { ws.set_spare("fold:", false); }
  ~FoldMemory() { ws_.set_spare("fold:", true); }
  cuapss_status or_probe(cuapss_status s, bool* done) {
    if (s != CUAPSS_ENOMEM) return s;
    *done = false;
    ws_.release_prefix("fold:");
    ws_.release_prefix("out:");
    return CUAPSS_OK;
  }

 private:
  Workspace& ws_;
};

}  // namespace

void note_fold(cuapss_ctx* ctx, bool mixed, const FoldResult* r) {
  for (int l = 0; l < kFoldLevels; ++l) {
    ctx->fold_columns[l] = r ? fold_k(mixed, l) : 0;
    ctx->fold_tiles[l] = r ? r->level_tiles[l] : 0;
  }
}

cuapss_status join_fold(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                        const int32_t* perm, double nrm2, const CostFn& other_ns, FoldResult* r,
                        bool* done) {
  *done = false;
  if (!verifiable(a) || (b && !verifiable(*b))) return CUAPSS_OK;
  FoldMemory mem(ctx->ws);
  return mem.or_probe(ctx->opts.precision == CUAPSS_PREC_MIXED
                          ? join_fold_as<true>(ctx, a, b, t, perm, nrm2, other_ns, r, done)
                          : join_fold_as<false>(ctx, a, b, t, perm, nrm2, other_ns, r, done),
                      done);
}

cuapss_status fold_batch(cuapss_ctx* ctx, const DevCsr& x, int k, const int64_t* inst_ptr,
                         const float* t, const int32_t* perm, double nrm2, double other_ns,
                         std::vector<int>* width, FoldResult* r, bool* done) {
  *done = false;
  if (!verifiable(x)) return CUAPSS_OK;
  FoldMemory mem(ctx->ws);
  return mem.or_probe(
      ctx->opts.precision == CUAPSS_PREC_MIXED
          ? fold_batch_as<true>(ctx, x, k, inst_ptr, t, perm, nrm2, other_ns, width, r, done)
          : fold_batch_as<false>(ctx, x, k, inst_ptr, t, perm, nrm2, other_ns, width, r, done),
      done);
}

cuapss_status fold_index(cuapss_ctx* ctx, bool mixed, const DevCsr& x, const int32_t* perm,
                         const FoldAlloc& alloc, FoldSide* s) {
  FoldMemory mem(ctx->ws);
  return mixed ? fold_index_as<true>(ctx, x, perm, alloc, s)
               : fold_index_as<false>(ctx, x, perm, alloc, s);
}

cuapss_status fold_query(cuapss_ctx* ctx, bool mixed, const std::vector<FoldSegment>& segs,
                         const DevCsr& q, const float* t, const float* t_row, const int32_t* perm,
                         double nrm2, double other_ns, int64_t rows, FoldResult* r, bool* done) {
  *done = false;
  if (!verifiable(q)) return CUAPSS_OK;
  for (const FoldSegment& g : segs)
    if (!verifiable(g.side->x)) return CUAPSS_OK;
  FoldMemory mem(ctx->ws);
  return mem.or_probe(
      mixed ? fold_query_as<true>(ctx, segs, q, t, t_row, perm, nrm2, other_ns, rows, r, done)
            : fold_query_as<false>(ctx, segs, q, t, t_row, perm, nrm2, other_ns, rows, r, done),
      done);
}

}  // namespace cuapss
