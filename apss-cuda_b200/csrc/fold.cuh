// Folded-bound join: a dense upper bound of every pair's similarity decides
// which pairs are computed at all.
//
// A row of K columns stands for a sparse row: the p = K / 4 most frequent
// features (frequency rank < p) keep a column each, and the other features
// share the remaining m = K - p columns, rank r in column p + (r - p) mod m,
// which holds the L2 norm of the row's values there. By Cauchy-Schwarz in
// every shared column,
//   s(a, b) <= sum_{k < p} a_k b_k + sum_{k >= p} A_k B_k,
// whatever the signs, so pairs whose folded dot product stays below t cannot
// be in the answer. The others (candidates) are computed in FP64 from the
// caller's CSR (verify.cu): the folding decides only what is looked at.
//
// The FP32 form keeps FP32 columns and products throughout.
//
// Rows are sorted by length, and the width K is chosen per pair of length
// classes from sampled rows (fold.cu): two short rows need few columns, two
// long ones many.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <functional>
#include <string>
#include <vector>

#include "common.cuh"
#include "ctx.cuh"

namespace cuapss {

// Lowest threshold of a folded join: its margins (about 0.01) stay small
// against t, and empty rows stay below it.
constexpr float kFoldMinT = 0.05f;

// Widths. Mixed precision: BF16 folds multiplied on the tensor cores, in
// 64-column chunks. FP32: FP32 folds multiplied on the CUDA cores, whose time
// is proportional to K (65 ns per column and 128 x 128 tile), so the widths
// are narrower and more candidates are computed.
constexpr int kFoldLevels = CUAPSS_FOLD_WIDTHS;
__host__ __device__ constexpr int fold_k(bool mixed, int level) {
  constexpr int k16[kFoldLevels] = {64, 128, 192, 256, 320, 384, 512, 768, 1024, 2048};
  constexpr int k32[kFoldLevels] = {16, 32, 48, 64, 96, 128, 192, 256, 512, 1024};
  return mixed ? k16[level] : k32[level];
}
// Columns per chunk (one bulk copy per chunk and row block), and the widest
// fold whose I chunks stay in shared memory.
constexpr int kFoldChunk16 = 64, kFoldResident16 = 256;
constexpr int kFoldChunk32 = 16, kFoldResident32 = 128;
constexpr int kFoldTileBytes = kBlockRows * kFoldChunk16 * 2;  // 16 KB
constexpr int kFoldSliceBytes = kBlockRows * kFoldChunk32 * 4;  // 8 KB

// One folded width of the two operands of a launch: [blocks][chunks], block
// `first` of the side at offset 0. BF16 chunks are 128 rows x 64 columns in
// the tensor cores' swizzled layout, FP32 chunks 16 columns x 128 rows.
struct FoldLevel {
  const uint8_t* I = nullptr;
  const uint8_t* J = nullptr;
  int firstI = 0, firstJ = 0;
  int nkc = 0;      // chunks
  float eps = 0.f;  // margin of the bound at this width
};

struct FoldTileArgs {
  FoldLevel lev[kFoldLevels];
  int64_t nI = 0, nJ = 0;
  int nbI = 0, nbJ = 0;
  int self = 0;                  // pairs i < j of one side only
  float t = 0.f;
  const float* t_row = nullptr;  // threshold of each J row, or null: t
  // Mixed: {I block, J0, J1, level | single << 7 | turn << 8}: blocks I and
  // I + 1 (single: I alone) x [J0, J1), from J0 + turn on, 0 <= turn < J1 - J0.
  const int4* units = nullptr;
  int nunits = 0;
  int* unit_counter = nullptr;
  uint64_t* cand = nullptr;      // {I row << 32 | J row}
  unsigned long long* cand_count = nullptr;
  int64_t cand_cap = 0;
  // > 0: a join with more candidates than this is given up. Once the list says
  // so, CTAs take no more units and warps list no more candidates.
  int64_t give_up_at = 0;
  int* err = nullptr;
  uint32_t* class_count = nullptr;  // sampling: [level][I block][J block] pairs at or above t - eps
};

// A unit's tiles in order, starting at J0 + turn and wrapping around, so that
// CTAs that work on the same J blocks at one time do not read the same L2
// lines in step (n = 200,000, K = 128: 993 -> 873 ns a tile when measured).
constexpr int kFoldSingle = 0x80;
struct FoldUnit {
  int I, J0, len, lev, turn;
  bool single;
  __device__ explicit FoldUnit(const int4& u)
      : I(u.x), J0(u.y), len(u.z - u.y), lev(u.w & 0x7f), turn(u.w >> 8),
        single((u.w & kFoldSingle) != 0) {}
  __device__ int J(int k) const {
    const int j = k + turn;
    return J0 + (j < len ? j : j - len);
  }
};

// count: adds to class_count instead of listing candidates. sms: SMs to fill.
cuapss_status launch_tiles_fold(const FoldTileArgs& a, int sms, cudaStream_t st, bool count);
// The FP32 form: units of one I block.
cuapss_status launch_tiles_fold32(const FoldTileArgs& a, int sms, cudaStream_t st, bool count);

constexpr int kFoldClasses = 16;  // length classes of a side

struct FoldOut {
  uint8_t* base[kFoldLevels] = {};  // null: not built
  int first[kFoldLevels] = {};      // block at offset 0
};

// One operand: its CSR, the order of its rows and its folded levels.
struct FoldSide {
  DevCsr x;
  int nb = 0;
  int64_t slots = 0;              // places, if some inside are empty (else x.n)
  int32_t* rowmap = nullptr;      // [128 nb] place -> caller's row, -1: empty
  const float* t_row = nullptr;   // per caller's row: rows are folded divided by it
  const float* t_place = nullptr; // per place: threshold of the row's products
  int edge[kFoldClasses + 1] = {};   // first block of each class (even), nb at the end
  double len[kFoldClasses] = {};     // mean row length of each class
  uint32_t levels[kFoldClasses];     // levels that may be used
  bool prepared = false;          // a resident index's side
  FoldOut out;
  int32_t* sample = nullptr;      // sampled rows, up to 128 per class
  FoldOut sample_out;
  FoldSide() {
    for (uint32_t& l : levels) l = (1u << kFoldLevels) - 1u;
  }
};

using FoldAlloc = std::function<cuapss_status(const std::string& name, size_t bytes, void** out)>;

// Exact decision of candidates (verify.cu).
struct VerifyArgs {
  const uint64_t* cand = nullptr;
  const unsigned long long* ncand = nullptr;  // device count (may exceed cap: nothing is done)
  int64_t cap = 0;
  unsigned* work = nullptr;  // group counter, zero at the launch
  const int32_t* permI = nullptr;  // place -> caller's row, or null: identity
  const int32_t* permJ = nullptr;
  const int64_t* rpI = nullptr;
  const int32_t* colI = nullptr;
  const float* valI = nullptr;
  const int64_t* rpJ = nullptr;
  const int32_t* colJ = nullptr;
  const float* valJ = nullptr;
  float t = 0.f;
  const float* t_row = nullptr;   // threshold of each J place, or
  const float* t_of_i = nullptr;  // of each of the I side's caller rows, or null: t
  int64_t j_offset = 0;              // added to the J row of every pair
  int self = 0;
  int rbits = 0;  // output key = (i << rbits) | j
  uint64_t* out_key = nullptr;
  uint32_t* out_idx = nullptr;
  float* out_sim = nullptr;
  unsigned long long* out_count = nullptr;
};
cuapss_status launch_verify(const VerifyArgs& a, cudaStream_t st);

// What a folded join did, for the statistics.
struct FoldResult {
  int64_t ncand = 0, npairs = 0, tiles = 0;
  uint64_t* okey = nullptr;  // unsorted output keys, payload indexes, similarities
  uint32_t* oidx = nullptr;
  float* osim = nullptr;
  int rbitsI = 1, rbitsJ = 1;
  double max_band = 0.0;  // widest margin of the widths used
  int64_t level_tiles[kFoldLevels] = {};  // 128 x 128 tiles multiplied at each width
};

// Records what the context's call did (null: it probed), for cuapss_fold_tiles.
void note_fold(cuapss_ctx* ctx, bool mixed, const FoldResult* r);

// Modelled cost, asked for only when it is needed.
using CostFn = std::function<cuapss_status(double* ns)>;

// The folded join of validated device matrices (b == nullptr: self-join), in
// the context's precision.
// *done = false: the probing path is the better one here and nothing was
// produced. other_ns: that path's modelled SM-nanoseconds per tile.
cuapss_status join_fold(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                        const int32_t* perm, double nrm2, const CostFn& other_ns, FoldResult* r,
                        bool* done);

// A resident index segment's side: order, levels and samples of x's rows,
// allocated through alloc.
cuapss_status fold_index(cuapss_ctx* ctx, bool mixed, const DevCsr& x, const int32_t* perm,
                         const FoldAlloc& alloc, FoldSide* s);

struct FoldSegment {
  FoldSide* side = nullptr;
  int64_t row0 = 0;
};

// The folded join of query rows (thresholds t on the host, t_row on the device)
// with the segments of an index of `rows` rows. *done and other_ns as in
// join_fold.
cuapss_status fold_query(cuapss_ctx* ctx, bool mixed, const std::vector<FoldSegment>& segs,
                         const DevCsr& q, const float* t, const float* t_row, const int32_t* perm,
                         double nrm2, double other_ns, int64_t rows, FoldResult* r, bool* done);

// The folded form of a batch of self-joins: instance q is the rows
// [inst_ptr[q], inst_ptr[q + 1]) of x at threshold t[q] (host arrays, all
// at least kFoldMinT). (*width)[q] receives the width of its folded rows (0: no
// pairs). *done and other_ns as in join_fold.
cuapss_status fold_batch(cuapss_ctx* ctx, const DevCsr& x, int k, const int64_t* inst_ptr,
                         const float* t, const int32_t* perm, double nrm2, double other_ns,
                         std::vector<int>* width, FoldResult* r, bool* done);

}  // namespace cuapss
