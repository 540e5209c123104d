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
constexpr int kClasses = 16;  // length classes of a side
// Upper edges of the classes as shares of the sorted rows: finer towards the
// long rows, whose folded products spread the most.
constexpr double kClassEdge[kClasses] = {0.125, 0.25, 0.375, 0.5,  0.625, 0.75,  0.8125, 0.875,
                                         0.92,  0.95, 0.97,  0.98, 0.988, 0.994, 0.998,  1.0};
// Sides of fewer blocks keep the caller's order and one width, whose
// candidates are few or, past kSmallMaxCand, make the join fall back.
constexpr int kSampleMinBlocks = 64;
constexpr int kSmallLevel = 3;
constexpr int64_t kSmallMaxCand = 1 << 21;

// Cost model, SM-nanoseconds, measured on 200,000 and 400,000 rows of the
// d = 50,000 workload. A 256 x 128 tile whose I chunks stay resident takes
// kTileNs + kChunkNs per 64 columns (K = 64: 616, 128: 873, 256: 1,446; the
// tensor cores alone 260 per 64 columns), a streamed one kStreamNs per 64
// columns (L2 bandwidth; K = 512: 3,212). A candidate takes kCandNs (its
// listing in the tile kernel, and verify) + kCandEntryNs per entry of its
// longer row.
constexpr double kTileNs = 340.0, kChunkNs = 275.0, kStreamNs = 400.0;
constexpr double kCandNs = 45.0, kCandEntryNs = 0.3;
// FP32, 128 x 128 tiles.
constexpr double kTile32Ns = 380.0, kColumn32Ns = 92.0;

template <bool MIXED>
constexpr int kPair = MIXED ? 2 : 1;  // I blocks of a tile
template <bool MIXED>
constexpr int kChunk = MIXED ? kFoldChunk16 : kFoldChunk32;

template <bool MIXED>
double tile_cost(int level) {
  const int K = fold_k(MIXED, level);
  if (!MIXED) return kTile32Ns + kColumn32Ns * K;
  return K <= kFoldResident16 ? kTileNs + kChunkNs * (K / 64) : kStreamNs * (K / 64);
}

template <bool MIXED>
cuapss_status launch_fold(const FoldTileArgs& a, int sms, cudaStream_t st, bool count) {
  return MIXED ? launch_tiles_fold(a, sms, st, count) : launch_tiles_fold32(a, sms, st, count);
}

inline unsigned grid_for(int64_t work, int per_block) {
  const int64_t g = ceil_div(std::max<int64_t>(work, 1), per_block);
  return (unsigned)std::min<int64_t>(g, 148 * 32);
}

// ---- row order: by length, in 256 classes of about 1/16 octave -----------
__global__ void k_len_keys(const int64_t* __restrict__ rp, int64_t n, uint64_t* __restrict__ keys,
                           uint32_t* __restrict__ vals) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float len = (float)(rp[i + 1] - rp[i]);
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
// memory (squares in the shared columns), in one pass over the row, and
// written as BF16 in the 128-byte-swizzled chunk layout of the tensor cores
// (prep.cu). Head values are rounded to nearest, which the margin covers;
// shared columns are rounded up after widening by the largest error their
// FP32 sums can have (2^-24 per addition), so their products bound the exact
// ones.
struct FoldOut {
  uint8_t* base[kFoldLevels];  // null: not built
  int first[kFoldLevels];      // block at offset 0
};

__host__ __device__ constexpr size_t fold_bytes(bool mixed, int level) {  // of a row block
  return (size_t)fold_k(mixed, level) * kBlockRows * (mixed ? 2 : 4);
}

// First accumulator column of level l when the levels of `allow` lie one
// after another, and their total.
__host__ __device__ constexpr int fold_offset(bool mixed, uint32_t allow, int l) {
  int o = 0;
  for (int k = 0; k < l; ++k)
    if ((allow >> k) & 1u) o += fold_k(mixed, k);
  return o;
}

template <bool MIXED, int LEV>
__device__ __forceinline__ void fold_add(uint32_t mask, float* acc, uint32_t allow, uint32_t r,
                                         float v) {
  constexpr uint32_t P = fold_k(MIXED, LEV) / 4, M = fold_k(MIXED, LEV) - P;
  if (!((mask >> LEV) & 1u)) return;  // uniform over the row's threads
  float* a = acc + fold_offset(MIXED, allow, LEV);
  if (r < P) a[r] = v;
  else atomicAdd(&a[P + (r - P) % M], v * v);
}

template <bool MIXED, int LEV>
__device__ __forceinline__ void fold_write(uint32_t mask, const float* acc, uint32_t allow,
                                           const FoldOut& O, float widen, int b, int rr, int tid,
                                           int nt) {
  constexpr int K = fold_k(MIXED, LEV), P = K / 4;
  if (!((mask >> LEV) & 1u)) return;
  const float* a = acc + fold_offset(MIXED, allow, LEV);
  uint8_t* dst = O.base[LEV] + (size_t)(b - O.first[LEV]) * fold_bytes(MIXED, LEV);
  if (!MIXED) {  // [column][row]
    for (int c = tid; c < K; c += nt)
      reinterpret_cast<float*>(dst)[c * kBlockRows + rr] =
          c < P ? a[c] : __fmul_ru(__fsqrt_ru(a[c]), widen);
    return;
  }
  uint4* out = reinterpret_cast<uint4*>(dst);
  for (int c8 = tid; c8 < K / 8; c8 += nt) {
    __nv_bfloat162 w[4];
    const float4 x = reinterpret_cast<const float4*>(a)[2 * c8];
    const float4 y = reinterpret_cast<const float4*>(a)[2 * c8 + 1];
    const float f[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (c8 * 8 < P) {  // P is a multiple of 8
        w[q].x = __float2bfloat16_rn(f[2 * q]);
        w[q].y = __float2bfloat16_rn(f[2 * q + 1]);
      } else {
        w[q].x = __float2bfloat16_ru(__fsqrt_ru(f[2 * q]) * widen);
        w[q].y = __float2bfloat16_ru(__fsqrt_ru(f[2 * q + 1]) * widen);
      }
    }
    const int kc = c8 >> 3, c = c8 & 7;
    uint4 u;
    memcpy(&u, w, 16);
    out[((size_t)kc * kBlockRows + rr) * 8 + (c ^ (rr & 7))] = u;
  }
}

// GROUP threads per row (a warp, or the whole CTA for long rows). Blocks
// [b0, b1) of rowmap; blk_mask[b]: levels of block b (null: mask0 for all);
// only blocks whose levels are all in `allow` (wide: some level is not
// narrow) are taken. Shared memory: the columns of `allow` per row.
constexpr uint32_t kNarrowLevels = 0x7f;  // K <= 512 (mixed), 192 (FP32)

template <bool MIXED, int GROUP>
__global__ void __launch_bounds__(kThreads)
    k_fold_rows(const int32_t* __restrict__ rowmap, int64_t slot0, int64_t slot1,
                const int64_t* __restrict__ rp, const int32_t* __restrict__ col,
                const float* __restrict__ val, const int32_t* __restrict__ perm,
                const uint16_t* __restrict__ blk_mask, uint32_t mask0, uint32_t allow, bool wide,
                FoldOut O) {
  extern __shared__ __align__(16) float fold_sm[];
  constexpr int kGroups = kThreads / GROUP;
  const int tid = threadIdx.x % GROUP;
  const int ncol = fold_offset(MIXED, allow, kFoldLevels);
  float* acc = fold_sm + (threadIdx.x / GROUP) * ncol;
  for (int64_t s = slot0 + (int64_t)blockIdx.x * kGroups + threadIdx.x / GROUP; s < slot1;
       s += (int64_t)gridDim.x * kGroups) {
    const int b = (int)(s / kBlockRows), rr = (int)(s % kBlockRows);
    const uint32_t mask = blk_mask ? (uint32_t)blk_mask[b] : mask0;
    if (mask == 0 || ((mask & ~kNarrowLevels) != 0) != wide) continue;  // same for all of GROUP
    const int32_t r = rowmap[s];
    const int64_t lo = r >= 0 ? rp[r] : 0;
    const int len = r >= 0 ? (int)(rp[r + 1] - lo) : 0;
    for (int k = tid; k < ncol / 4; k += GROUP)
      reinterpret_cast<float4*>(acc)[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (GROUP == 32) __syncwarp();
    else __syncthreads();
    for (int e = tid; e < len; e += GROUP) {
      const uint32_t f = (uint32_t)perm[col[lo + e]];
      const float v = val[lo + e];
      fold_add<MIXED, 0>(mask, acc, allow, f, v);
      fold_add<MIXED, 1>(mask, acc, allow, f, v);
      fold_add<MIXED, 2>(mask, acc, allow, f, v);
      fold_add<MIXED, 3>(mask, acc, allow, f, v);
      fold_add<MIXED, 4>(mask, acc, allow, f, v);
      fold_add<MIXED, 5>(mask, acc, allow, f, v);
      fold_add<MIXED, 6>(mask, acc, allow, f, v);
      fold_add<MIXED, 7>(mask, acc, allow, f, v);
      fold_add<MIXED, 8>(mask, acc, allow, f, v);
      fold_add<MIXED, 9>(mask, acc, allow, f, v);
    }
    if (GROUP == 32) __syncwarp();
    else __syncthreads();
    const float widen = 1.0f + (float)(len + 16) * 5.9604645e-8f * 1.01f;
    fold_write<MIXED, 0>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 1>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 2>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 3>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 4>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 5>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 6>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 7>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 8>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    fold_write<MIXED, 9>(mask, acc, allow, O, widen, b, rr, tid, GROUP);
    if (GROUP == 32) __syncwarp();
    else __syncthreads();
  }
}
static_assert(kFoldLevels == 10, "one fold_add / fold_write call per level");

// Folds the places of [0, slots) with the levels of masks (host, per block;
// empty: mask0 everywhere) into O.
template <bool MIXED>
cuapss_status fold_side(const DevCsr& x, const int32_t* rowmap, int64_t slots,
                        const std::vector<uint16_t>& masks, uint32_t mask0, const int32_t* perm,
                        const FoldOut& O, Workspace& ws, const std::string& tag, cudaStream_t st) {
  uint16_t* d_mask = nullptr;
  // levels, and blocks, with and without a wide level
  uint32_t all[2] = {0, 0};
  int64_t b0[2] = {0, 0}, b1[2] = {0, 0};
  if (masks.empty()) {
    const int w = (mask0 & ~kNarrowLevels) ? 1 : 0;
    all[w] = mask0;
    b1[w] = slots / kBlockRows;
  } else {
    ST_TRY(ws.get(tag + ":mask", masks.size(), &d_mask));
    CU_TRY(cudaMemcpyAsync(d_mask, masks.data(), 2 * masks.size(), cudaMemcpyHostToDevice, st));
    for (size_t b = 0; b < masks.size(); ++b) {
      const int w = (masks[b] & ~kNarrowLevels) ? 1 : 0;
      if (!all[w]) b0[w] = (int64_t)b;
      all[w] |= masks[b];
      if (masks[b]) b1[w] = (int64_t)b + 1;
    }
  }
  if (all[0]) {  // a warp per row
    const size_t smem = (size_t)fold_offset(MIXED, all[0], kFoldLevels) * 4 * (kThreads / 32);
    CU_TRY(cudaFuncSetAttribute((const void*)k_fold_rows<MIXED, 32>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                fold_offset(MIXED, kNarrowLevels, kFoldLevels) * 4 *
                                    (kThreads / 32)));
    k_fold_rows<MIXED, 32><<<grid_for((b1[0] - b0[0]) * kBlockRows, kThreads / 32), kThreads, smem, st>>>(
        rowmap, b0[0] * kBlockRows, b1[0] * kBlockRows, x.rp, x.col, x.val, perm, d_mask, mask0,
        all[0], false, O);
    LAUNCH_CHECK();
  }
  if (all[1]) {  // blocks of long rows (and the samples): a CTA per row
    const size_t smem = (size_t)fold_offset(MIXED, all[1], kFoldLevels) * 4;
    k_fold_rows<MIXED, kThreads><<<grid_for((b1[1] - b0[1]) * kBlockRows, 1), kThreads, smem, st>>>(
        rowmap, b0[1] * kBlockRows, b1[1] * kBlockRows, x.rp, x.col, x.val, perm, d_mask, mask0,
        all[1], true, O);
    LAUNCH_CHECK();
  }
  return CUAPSS_OK;
}

float fold_eps(bool mixed, int level, double nrm2) {
  // mixed: BF16 rounding of the head columns, FP32 accumulation of K / 16
  // steps; FP32: a chain of K FMAs
  const int K = fold_k(mixed, level);
  const double head = mixed ? std::ldexp(1.0, -7) + std::ldexp(1.0, -16) : 0.0;
  const double acc =
      (mixed ? (K / 16.0 + 2.0) * std::ldexp(1.0, -20) : (K + 4.0) * std::ldexp(1.0, -24)) * 1.02;
  return (float)((head + acc) * nrm2 * 1.001 + 1e-6);
}

struct FoldSide {
  DevCsr x;
  int nb = 0;
  int32_t* rowmap = nullptr;      // [128 nb] place -> caller's row, -1 past n
  int edge[kClasses + 1] = {};    // first block of each class (even), nb at the end
  double len[kClasses] = {};      // mean row length of each class
  int32_t* sample = nullptr;
  std::vector<uint16_t> masks;     // levels of each block
  FoldOut out{};
};

// Row order and class edges.
cuapss_status order_side(FoldSide& s, bool by_length, Workspace& ws, const std::string& tag,
                         cudaStream_t st) {
  s.nb = (int)ceil_div(s.x.n, kBlockRows);
  const int64_t slots = (int64_t)s.nb * kBlockRows;
  ST_TRY(ws.get(tag + ":map", (size_t)slots, &s.rowmap));
  uint32_t* vals = nullptr;
  if (by_length) {
    uint64_t* keys = nullptr;
    ST_TRY(ws.get(tag + ":keys", (size_t)s.x.n, &keys));
    ST_TRY(ws.get(tag + ":vals", (size_t)s.x.n, &vals));
    k_len_keys<<<grid_for(s.x.n, kThreads), kThreads, 0, st>>>(s.x.rp, s.x.n, keys, vals);
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

// The width of every pair of classes, from the products of sampled rows.
// level[a][b] (I class a, J class b; self: b >= a) and the modelled cost of
// the join in SM-nanoseconds, with its expected candidates.
template <bool MIXED>
cuapss_status plan_levels(cuapss_ctx* ctx, FoldSide& I, FoldSide& J, bool self, float t,
                          const int32_t* perm, double nrm2, int (*level)[kClasses], double* cost,
                          double* cands) {
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  const int64_t slots = (int64_t)kClasses * kBlockRows;
  const size_t ncnt = (size_t)kFoldLevels * kClasses * kClasses;
  unsigned long long* stats = nullptr;  // row length sums, then pair counts
  ST_TRY(ws.get("fold:stats", 2 * kClasses + ncnt / 2, &stats));
  uint32_t* cnt = reinterpret_cast<uint32_t*>(stats + 2 * kClasses);
  CU_TRY(cudaMemsetAsync(stats, 0, 8 * (2 * kClasses) + 4 * ncnt, st));
  FoldTileArgs ta;
  FoldSide* side[2] = {&I, &J};
  for (int k = 0; k < (self ? 1 : 2); ++k) {
    FoldSide& s = *side[k];
    const std::string tag = k == 0 ? "fold:sI" : "fold:sJ";
    ST_TRY(ws.get(tag, (size_t)slots, &s.sample));
    k_sample_rows<<<kClasses, kBlockRows, 0, st>>>(s.rowmap, s.x.rp, class_rows(s), s.sample,
                                                   stats + k * kClasses);
    LAUNCH_CHECK();
    FoldOut o{};
    for (int l = 0; l < kFoldLevels; ++l)
      ST_TRY(ws.get(tag + std::to_string(l), kClasses * fold_bytes(MIXED, l), &o.base[l]));
    ST_TRY(fold_side<MIXED>(s.x, s.sample, slots, {}, (1u << kFoldLevels) - 1u, perm, o, ws, tag, st));
    for (int l = 0; l < kFoldLevels; ++l) {
      if (k == 0) ta.lev[l].I = o.base[l];
      if (k == 1 || self) ta.lev[l].J = o.base[l];
    }
  }
  std::vector<int4> units;
  for (int l = kFoldLevels - 1; l >= 0; --l) {
    ta.lev[l].nkc = fold_k(MIXED, l) / kChunk<MIXED>;
    ta.lev[l].eps = fold_eps(MIXED, l, nrm2);
    for (int a = 0; a < kClasses; a += kPair<MIXED>)
      for (int b = self ? a : 0; b < kClasses; ++b) units.push_back(make_int4(a, b, b + 1, l));
  }
  int4* d_units = nullptr;
  int* ctl = nullptr;
  ST_TRY(ws.get("fold:sunits", units.size(), &d_units));
  ST_TRY(ws.get("fold:sctl", 2, &ctl));
  CU_TRY(cudaMemcpyAsync(d_units, units.data(), sizeof(int4) * units.size(),
                         cudaMemcpyHostToDevice, st));
  CU_TRY(cudaMemsetAsync(ctl, 0, 2 * sizeof(int), st));
  ta.nI = ta.nJ = slots;
  ta.nbI = ta.nbJ = kClasses;
  ta.t = t;
  ta.units = d_units;
  ta.nunits = (int)units.size();
  ta.unit_counter = ctl;
  ta.err = ctl + 1;
  ta.class_count = cnt;
  ST_TRY(launch_fold<MIXED>(ta, ctx->sms, st, true));
  std::vector<uint8_t> h(8 * 2 * kClasses + 4 * ncnt);
  int herr = 0;
  CU_TRY(cudaMemcpyAsync(h.data(), stats, h.size(), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaMemcpyAsync(&herr, ctl + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
  CU_TRY(cudaStreamSynchronize(st));
  if (herr & kErrTimeout) return CUAPSS_ETIMEOUT;
  if (herr) return CUAPSS_ECUDA;
  const unsigned long long* hl = reinterpret_cast<const unsigned long long*>(h.data());
  const uint32_t* hc = reinterpret_cast<const uint32_t*>(hl + 2 * kClasses);
  ClassRows cr[2] = {class_rows(I), class_rows(J)};
  double rows[2][kClasses];
  for (int k = 0; k < 2; ++k)
    for (int c = 0; c < kClasses; ++c) {
      rows[k][c] = (double)std::min<int64_t>(kBlockRows, cr[k].row[c + 1] - cr[k].row[c]);
      const int src = self ? 0 : k;
      side[k]->len[c] = rows[k][c] > 0 ? (double)hl[src * kClasses + c] / rows[k][c] : 0.0;
    }
  *cost = *cands = 0.0;
  for (int a = 0; a < kClasses; ++a)
    for (int b = self ? a : 0; b < kClasses; ++b) {
      const double sampled = rows[0][a] * rows[1][b] - (self && a == b ? rows[0][a] : 0.0);
      const double nI = (double)(cr[0].row[a + 1] - cr[0].row[a]);
      const double nJ = (double)(cr[1].row[b + 1] - cr[1].row[b]);
      const double pairs = self && a == b ? nI * (nI - 1) / 2 : nI * nJ;
      double best = 1e300, best_cand = 0.0;
      level[a][b] = 0;
      for (int l = 0; l < kFoldLevels; ++l) {
        double c = (double)hc[((size_t)l * kClasses + a) * kClasses + b];
        if (self && a == b) c = std::max(0.0, c - rows[0][a]);  // a row with itself
        // a count of zero is not a share of zero: half a pair
        const double share = sampled > 0 ? std::max(c, 0.5) / sampled : 0.0;
        const double tiles = pairs / ((double)kPair<MIXED> * kBlockRows * kBlockRows);
        const double cand_ns =
            kCandNs + kCandEntryNs * std::max(side[0]->len[a], side[1]->len[b]);
        const double ns = tiles * tile_cost<MIXED>(l) + share * pairs * cand_ns;
        if (ns < best) {
          best = ns;
          best_cand = share * pairs;
          level[a][b] = l;
        }
      }
      *cost += best;
      *cands += best_cand;
    }
  return CUAPSS_OK;
}

int class_of(const FoldSide& s, int block) {
  int c = 0;
  while (c + 1 < kClasses && block >= s.edge[c + 1]) ++c;
  return c;
}

// Allocates and builds the folded levels a side needs.
template <bool MIXED>
cuapss_status build_levels(FoldSide& s, const uint32_t (&need)[kClasses], const int32_t* perm,
                           Workspace& ws, const std::string& tag, cudaStream_t st) {
  uint32_t all = 0;
  for (int c = 0; c < kClasses; ++c)
    if (s.edge[c + 1] > s.edge[c]) all |= need[c];
  for (int l = 0; l < kFoldLevels; ++l) {
    if (!((all >> l) & 1u)) continue;
    int lo = s.nb, hi = 0;
    for (int c = 0; c < kClasses; ++c)
      if (s.edge[c + 1] > s.edge[c] && ((need[c] >> l) & 1u)) {
        lo = std::min(lo, s.edge[c]);
        hi = std::max(hi, s.edge[c + 1]);
      }
    s.out.first[l] = lo;
    ST_TRY(ws.get(tag + ":lev" + std::to_string(l), (size_t)(hi - lo) * fold_bytes(MIXED, l),
                  &s.out.base[l]));
  }
  s.masks.assign((size_t)s.nb, 0);
  for (int c = 0; c < kClasses; ++c)
    for (int b = s.edge[c]; b < s.edge[c + 1]; ++b) s.masks[(size_t)b] = (uint16_t)need[c];
  return fold_side<MIXED>(s.x, s.rowmap, (int64_t)s.nb * kBlockRows, s.masks, 0, perm, s.out, ws,
                          tag, st);
}

// Units: windows of J blocks from the long rows down (the costly units
// first), in each window every I pair against each class's part of it, so
// that the CTAs running at one time share a window's chunks in L2. Wider
// folds get proportionally shorter ranges.
template <bool MIXED>
void make_units(const FoldSide& I, const FoldSide& J, bool self, const int (*level)[kClasses],
                int sms, std::vector<int4>* units, int64_t* tiles) {
  const int nbJ = J.nb;
  const int pair = kPair<MIXED>;
  const double total = (self ? 0.5 * nbJ * (nbJ + 2.0) : (double)I.nb * nbJ) / pair;
  const int w = (int)std::max(1.0, std::min(MIXED ? 128.0 : 32.0, total / (sms * 16.0)));
  for (int j1 = nbJ; j1 > 0; j1 -= w) {
    const int j0 = std::max(0, j1 - w);
    for (int b = class_of(J, j1 - 1); b >= 0 && J.edge[b + 1] > j0; --b) {
      const int s0 = std::max(j0, J.edge[b]), s1 = std::min(j1, J.edge[b + 1]);
      if (s0 >= s1) continue;
      int a = 0;
      for (int i = 0; i < (self ? std::min(I.nb, s1) : I.nb); i += pair) {
        while (i >= I.edge[a + 1]) ++a;
        const int lv = level[a][b];
        const int f0 = self ? std::max(s0, i) : s0;
        const double rel = tile_cost<MIXED>(lv) / tile_cost<MIXED>(MIXED ? 1 : 3);
        const int step = std::max(1, (int)(w / std::max(1.0, rel)));
        for (int f = f0; f < s1; f += step) {
          const int len = std::min(s1 - f, step);
          // spread the starts of neighbouring units over the range
          const int turn = (int)(((int64_t)(units->size() % 16) * len) / 16);
          units->push_back(make_int4(i, f, f + len, lv | turn << 8));
        }
      }
    }
  }
  *tiles = self ? (int64_t)nbJ * (nbJ + 1) / 2 : (int64_t)I.nb * nbJ;
}

template <bool MIXED>
cuapss_status join_fold_as(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                           const int32_t* perm, double nrm2, double other_ns, FoldResult* r,
                           bool* done) {
  *done = false;
  const bool self = b == nullptr;
  Workspace& ws = ctx->ws;
  cudaStream_t st = ctx->stream;
  FoldSide SI, SJ;
  SI.x = a;
  if (!self) SJ.x = *b;
  FoldSide& J = self ? SI : SJ;
  const int64_t nbI = ceil_div(SI.x.n, kBlockRows), nbJ = ceil_div(J.x.n, kBlockRows);
  const double tiles128 = self ? 0.5 * nbI * (nbI + 1.0) : (double)nbI * nbJ;
  const bool sampled = tiles128 >= 0.5 * kSampleMinBlocks * kSampleMinBlocks;
  ST_TRY(order_side(SI, sampled, ws, "fold:I", st));
  if (!self) ST_TRY(order_side(SJ, sampled, ws, "fold:J", st));
  int level[kClasses][kClasses];
  double cands = 0.0;
  if (sampled) {
    double cost = 0.0;
    ST_TRY(plan_levels<MIXED>(ctx, SI, J, self, t, perm, nrm2, level, &cost, &cands));
    if (cost >= tiles128 * other_ns) return CUAPSS_OK;
  } else {
    for (auto& row : level)
      for (int& l : row) l = kSmallLevel;  // K = 256 or 64
  }
  // ---- folded operands
  uint32_t needI[kClasses] = {}, needJ[kClasses] = {};
  for (int x = 0; x < kClasses; ++x)
    for (int y = self ? x : 0; y < kClasses; ++y) {
      if (SI.edge[x + 1] <= SI.edge[x] || J.edge[y + 1] <= J.edge[y]) continue;
      needI[x] |= 1u << level[x][y];
      needJ[y] |= 1u << level[x][y];
    }
  if (self)
    for (int c = 0; c < kClasses; ++c) needI[c] |= needJ[c];
  ST_TRY(build_levels<MIXED>(SI, needI, perm, ws, "fold:I", st));
  if (!self) ST_TRY(build_levels<MIXED>(SJ, needJ, perm, ws, "fold:J", st));
  // ---- units
  std::vector<int4> units;
  make_units<MIXED>(SI, J, self, level, ctx->sms, &units, &r->tiles);
  int4* d_units = nullptr;
  ST_TRY(ws.get("tiles:units", std::max<size_t>(units.size(), 1), &d_units));
  if (!units.empty())
    CU_TRY(cudaMemcpyAsync(d_units, units.data(), sizeof(int4) * units.size(),
                           cudaMemcpyHostToDevice, st));
  // control words: candidates, pairs found, {unit counter, verify's group
  // counter}, error flags
  unsigned long long* ctl = nullptr;
  ST_TRY(ws.get("fold:ctl", 4, &ctl));
  FoldTileArgs ta;
  for (int l = 0; l < kFoldLevels; ++l) {
    FoldLevel& L = ta.lev[l];
    L.I = SI.out.base[l];
    L.J = J.out.base[l];
    L.firstI = SI.out.first[l];
    L.firstJ = J.out.first[l];
    L.nkc = fold_k(MIXED, l) / kChunk<MIXED>;
    L.eps = fold_eps(MIXED, l, nrm2);
    if (SI.out.base[l]) r->max_band = std::max(r->max_band, (double)L.eps);
  }
  ta.nI = SI.x.n;
  ta.nJ = J.x.n;
  ta.nbI = SI.nb;
  ta.nbJ = J.nb;
  ta.self = self ? 1 : 0;
  ta.t = t;
  ta.units = d_units;
  ta.nunits = (int)units.size();
  ta.cand_count = ctl;
  ta.unit_counter = reinterpret_cast<int*>(ctl + 2);
  ta.err = reinterpret_cast<int*>(ctl + 3);
  r->rbitsI = std::max(1, bits_for((uint64_t)SI.x.n));
  r->rbitsJ = std::max(1, bits_for((uint64_t)J.x.n));
  VerifyArgs va;
  va.permI = SI.rowmap;
  va.permJ = J.rowmap;
  va.rpI = SI.x.rp;
  va.colI = SI.x.col;
  va.valI = SI.x.val;
  va.rpJ = J.x.rp;
  va.colJ = J.x.col;
  va.valJ = J.x.val;
  va.t = t;
  va.self = ta.self;
  va.rbits = r->rbitsJ;
  va.ncand = ctl;
  va.out_count = ctl + 1;
  va.work = reinterpret_cast<unsigned*>(ctl + 2) + 1;
  int64_t cap = std::max<int64_t>(sampled ? (int64_t)(1.5 * cands) : 0,
                                  std::max<int64_t>(1 << 20, SI.x.n + J.x.n));
  for (int attempt = 0; attempt < 3; ++attempt) {
    ST_TRY(ws.get("fold:cand", (size_t)cap, &ta.cand));
    ST_TRY(ws.get("out:key", (size_t)cap, &r->okey));
    ST_TRY(ws.get("out:idx", (size_t)cap, &r->oidx));
    ST_TRY(ws.get("out:sim", (size_t)cap, &r->osim));
    ta.cand_cap = cap;
    CU_TRY(cudaMemsetAsync(ctl, 0, 4 * sizeof(unsigned long long), st));
    ST_TRY(launch_fold<MIXED>(ta, ctx->sms, st, false));
    va.cand = ta.cand;
    va.cap = cap;
    va.out_key = r->okey;
    va.out_idx = r->oidx;
    va.out_sim = r->osim;
    ST_TRY(launch_verify(va, st));
    unsigned long long h[4] = {0, 0, 0, 0};
    CU_TRY(cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    if (h[3] & kErrTimeout) return CUAPSS_ETIMEOUT;
    if (h[3]) return CUAPSS_ECUDA;
    r->ncand = (int64_t)h[0];
    r->npairs = (int64_t)h[1];
    if (r->ncand <= cap) {
      *done = true;
      return CUAPSS_OK;
    }
    // an unsampled join that the bound does not prune, or one whose sample
    // misjudged it: the probing path takes it
    if (r->ncand > (sampled ? 4 * cap : kSmallMaxCand)) return CUAPSS_OK;
    cap = r->ncand;
  }
  return CUAPSS_OK;
}

}  // namespace

cuapss_status join_fold(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                        const int32_t* perm, double nrm2, double other_ns, FoldResult* r,
                        bool* done) {
  return ctx->opts.precision == CUAPSS_PREC_MIXED
             ? join_fold_as<true>(ctx, a, b, t, perm, nrm2, other_ns, r, done)
             : join_fold_as<false>(ctx, a, b, t, perm, nrm2, other_ns, r, done);
}

}  // namespace cuapss
