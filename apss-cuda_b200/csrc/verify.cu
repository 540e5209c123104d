// Exact decision of the folded join's candidates: every candidate's
// similarity in FP64 from the caller's CSR, kept if >= t.
//
// A warp takes up to 32 consecutive candidates: their row numbers and row
// pointers load one candidate per lane, then the warp computes them in turn,
// the lanes running over the shorter row and searching the longer one. The
// sum's order differs from the oracle's ascending feature order, so a sum
// within the FP64 rounding of t is redone in that order by one lane; every
// decision is then the oracle's. The order depends on the two rows alone, so
// a pair's value does not depend on how the join was cut.
//
// Bound: latency of the searches' loads (rows come from L2), hidden by 64
// warps a SM.
#include <cuda_runtime.h>

#include "fold.cuh"

namespace cuapss {

namespace {

constexpr int kThreads = 256;
constexpr unsigned kFull = 0xffffffffu;

// FP64 merge-dot over two rows sorted by feature id (the oracle's order).
__device__ double dot_ordered(const int32_t* __restrict__ ca, const float* __restrict__ va, int na,
                              const int32_t* __restrict__ cb, const float* __restrict__ vb, int nb) {
  double s = 0.0;
  int a = 0, b = 0;
  while (a < na && b < nb) {
    const int32_t x = ca[a], y = cb[b];
    if (x == y) s = __dadd_rn(s, __dmul_rn((double)va[a], (double)vb[b]));
    a += x <= y;
    b += y <= x;
  }
  return s;
}

__global__ void __launch_bounds__(kThreads) k_verify(const VerifyArgs A) {
  const int64_t nc = (int64_t)*A.ncand;
  if (nc > A.cap) return;  // incomplete list: the host runs again with room
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t wid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int g = 32;  // candidates a warp takes at a time: fewer when there are few
  while (g > 1 && (int64_t)g * warps > nc) g >>= 1;
  for (int64_t base = wid * g; base < nc; base += warps * g) {
    const int m = (int)(nc - base < g ? nc - base : g);
    uint32_t pi = 0, pj = 0;  // caller's rows
    uint32_t so = 0, lo = 0;  // first entry of the shorter and the longer row
    int sl = 0, ll = 0;       // their lengths
    bool swapped = false;     // the shorter row is J's
    double t = 0.0;
    if (lane < m) {
      const uint64_t key = A.cand[base + lane];
      const uint32_t ip = (uint32_t)(key >> 32), jp = (uint32_t)key;
      t = A.t_row ? (double)A.t_row[jp] : (double)A.t;
      pi = A.permI ? (uint32_t)A.permI[ip] : ip;
      pj = A.permJ ? (uint32_t)A.permJ[jp] : jp;
      const int64_t a0 = A.rpI[pi], b0 = A.rpJ[pj];
      const int na = (int)(A.rpI[pi + 1] - a0), nb = (int)(A.rpJ[pj + 1] - b0);
      // equal lengths: the smaller row number of a self-join leads
      swapped = nb < na || (nb == na && A.self && pj < pi);
      so = (uint32_t)(swapped ? b0 : a0);
      lo = (uint32_t)(swapped ? a0 : b0);
      sl = swapped ? nb : na;
      ll = swapped ? na : nb;
    }
    double mine = 0.0;
    for (int k = 0; k < m; ++k) {
      const uint32_t so_k = __shfl_sync(kFull, so, k), lo_k = __shfl_sync(kFull, lo, k);
      const int sl_k = __shfl_sync(kFull, sl, k), ll_k = __shfl_sync(kFull, ll, k);
      const bool sw_k = __shfl_sync(kFull, (int)swapped, k) != 0;
      const int32_t* __restrict__ cs = (sw_k ? A.colJ : A.colI) + so_k;
      const float* __restrict__ vs = (sw_k ? A.valJ : A.valI) + so_k;
      const int32_t* __restrict__ cl = (sw_k ? A.colI : A.colJ) + lo_k;
      const float* __restrict__ vl = (sw_k ? A.valI : A.valJ) + lo_k;
      double s = 0.0;
      for (int e = lane; e < sl_k; e += 32) {
        const int32_t c = cs[e];
        int x = 0, n = ll_k;  // lower bound of c in cl
        while (n > 0) {
          const int h = n >> 1;
          const bool right = cl[x + h] < c;
          x = right ? x + h + 1 : x;
          n = right ? n - h - 1 : h;
        }
        if (x < ll_k && cl[x] == c) s += (double)vs[e] * (double)vl[x];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
      if (lane == k) mine = s;
    }
    bool in = false;
    if (lane < m) {
      // two orders of at most sl products of a sum near t <= 2 differ by less
      // than sl 2^-51 (all partial sums are at most the norms' product, < 2)
      if (fabs(mine - t) <= (double)(sl + 4) * 8.9e-16) {
        mine = dot_ordered((swapped ? A.colJ : A.colI) + so, (swapped ? A.valJ : A.valI) + so, sl,
                           (swapped ? A.colI : A.colJ) + lo, (swapped ? A.valI : A.valJ) + lo, ll);
      }
      in = mine >= t;
    }
    const unsigned found = __ballot_sync(kFull, in);
    if (!found) continue;
    unsigned long long w = 0;
    if (lane == 0) w = atomicAdd(A.out_count, (unsigned long long)__popc(found));
    w = __shfl_sync(kFull, w, 0) + (unsigned long long)__popc(found & ((1u << lane) - 1u));
    if (in) {  // w < nc <= cap
      uint64_t x = pi, y = pj;
      if (A.self && x > y) {
        x = pj;
        y = pi;
      }
      A.out_key[w] = (x << A.rbits) | y;
      A.out_idx[w] = (uint32_t)w;
      A.out_sim[w] = (float)mine;
    }
  }
}

}  // namespace

cuapss_status launch_verify(const VerifyArgs& a, cudaStream_t st) {
  k_verify<<<148 * 8, kThreads, 0, st>>>(a);
  LAUNCH_CHECK();
  return CUAPSS_OK;
}

}  // namespace cuapss
