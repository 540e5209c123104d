// Context object behind the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <string>
#include <vector>

#include "common.cuh"
#include "cuapss.h"
#include "prep.cuh"
#include "side.cuh"

struct cuapss_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  cuapss_opts opts{};
  int sms = 148;
  cuapss::Workspace ws;
  cudaEvent_t ev[6] = {};
  int64_t cand_cap = 0;
  void* pinned = nullptr;  // kPinnedBytes of host memory for small copies back
  // folded 128 x 128 tiles of the last call by width (columns 0: none)
  int32_t fold_columns[CUAPSS_FOLD_WIDTHS] = {};
  int64_t fold_tiles[CUAPSS_FOLD_WIDTHS] = {};
  // batched joins: the captured tile launches (updated in place when the
  // next batch has the same launch topology) and the tuner's choices
  cudaGraph_t batch_graph = nullptr;
  cudaGraphExec_t batch_exec = nullptr;
  std::map<uint64_t, int> tuned_p;
};

namespace cuapss {

constexpr size_t kPinnedBytes = 64 * 1024;

struct DevCsr {
  int64_t n = 0, d = 0, nnz = 0;
  const int64_t* rp = nullptr;
  const int32_t* col = nullptr;
  const float* val = nullptr;
  bool nonneg = false;  // no value is negative (known after validation)
};

// Validates the descriptor and returns device pointers (staging host
// arrays into workspace buffers named by tag).
cuapss_status stage_csr(cuapss_ctx* ctx, const cuapss_csr* x, const std::string& tag,
                        DevCsr* out);

// The self-join (b == nullptr) or cross-join of staged matrices.
cuapss_status join_device(cuapss_ctx* ctx, const DevCsr& a, const DevCsr* b, float t,
                          cuapss_pairs* out, cuapss_stats* stats, int shard = 0,
                          int nshards = 1);

// Sorts npairs unsorted output pairs (keys (i << rbitsJ) | j of keybits bits,
// payload indexes into sim) and writes them to out: CUAPSS_EOVERFLOW, with
// the count set, when its capacity is too small.
cuapss_status emit_pairs(cuapss_ctx* ctx, uint64_t* key, uint32_t* idx, const float* sim,
                         int64_t npairs, int keybits, int rbitsJ, cuapss_pairs* out);

// Head width used when the options leave it to the library: n rows, nnz
// non-zeros over d features; prefix[k] = postings of the k most frequent
// features (rank_count_prefix; may be empty for FP32). Self-joins whose rare
// features are paired explicitly pass the first rank of those features and
// their postings (0: every tail feature is probed).
int choose_head_width(int precision, int64_t n, int64_t d, int64_t nnz,
                      const std::vector<int64_t>& prefix, int64_t rare_rank = 0,
                      int64_t rare_postings = 0);

// Whether the tile cost model puts the head at p at least twice the tail
// still probed (the tile kernel's two-J-block MMA tiles then pay).
bool head_bound_plan(int64_t p, int64_t n, int64_t nnz, const std::vector<int64_t>& prefix,
                     const RareCandidate& rare);

// Head width and rare-feature threshold of a self-join, chosen together by
// the tile cost model: the threshold (of cands, at most max_pairs pairs, or
// none) and p that minimise the modelled tile time plus the explicit pairs'
// cost. fixed_p > 0: that head width, the threshold alone is chosen.
// forced: the (single) candidate is taken whatever its modelled cost.
struct TilePlan {
  int p = 0;
  RareCandidate rare;  // max_count 0: no explicit pairs
  double tile_ns = 0.0;  // modelled SM-nanoseconds of one tile, explicit pairs included
};
TilePlan plan_tiles(int precision, int64_t n, int64_t d, int64_t nnz,
                    const std::vector<int64_t>& prefix,
                    const std::vector<RareCandidate>& cands, int64_t max_pairs, int fixed_p,
                    bool forced = false);

// Modelled SM-nanoseconds of an FP32 probing tile of rows with nnz / n
// non-zeros each.
double plain_tile_ns(int64_t nnz, int64_t n);

}  // namespace cuapss
