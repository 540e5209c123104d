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
// Rows are sorted by length, and the width K is chosen per pair of length
// classes from sampled rows (fold.cu): two short rows need few columns, two
// long ones many.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "common.cuh"
#include "ctx.cuh"

namespace cuapss {

constexpr int kFoldLevels = 8;
constexpr int kFoldK[kFoldLevels] = {64, 128, 192, 256, 384, 512, 1024, 2048};
constexpr int kFoldResidentK = 256;  // widest fold whose I chunks stay in shared memory
constexpr int kFoldTileBytes = kBlockRows * 64 * 2;  // a 64-column BF16 chunk of a row block

// One folded width of the two operands of a launch: [blocks][K / 64] chunks
// of 16 KB, block `first` of the side at offset 0.
struct FoldLevel {
  const uint8_t* I = nullptr;
  const uint8_t* J = nullptr;
  int firstI = 0, firstJ = 0;
  int nkc = 0;      // K / 64
  float eps = 0.f;  // margin of the bound at this width
};

struct FoldTileArgs {
  FoldLevel lev[kFoldLevels];
  int64_t nI = 0, nJ = 0;
  int nbI = 0, nbJ = 0;
  int self = 0;                  // pairs i < j of one side only
  float t = 0.f;
  const float* t_row = nullptr;  // threshold of each J row, or null: t
  const int4* units = nullptr;   // {I block (even), J0, J1, level | turn << 8}: blocks I, I + 1 x
                                 // [J0, J1), from J0 + turn on (0 <= turn < J1 - J0)
  int nunits = 0;
  int* unit_counter = nullptr;
  uint64_t* cand = nullptr;      // {I row << 32 | J row}
  unsigned long long* cand_count = nullptr;
  int64_t cand_cap = 0;
  int* err = nullptr;
  uint32_t* class_count = nullptr;  // sampling: [level][I block][J block] pairs at or above t - eps
};

// count: adds to class_count instead of listing candidates.
cuapss_status launch_tiles_fold(const FoldTileArgs& a, int grid, cudaStream_t st, bool count);

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
  const float* t_row = nullptr;  // threshold of each J place, or null: t
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
};

// The folded join of validated device matrices (b == nullptr: self-join).
// *done = false: the probing path is the better one here and nothing was
// produced. other_ns: that path's modelled SM-nanoseconds per tile.
cuapss_status join_fold(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                        const int32_t* perm, double nrm2, double other_ns, FoldResult* r,
                        bool* done);

}  // namespace cuapss
