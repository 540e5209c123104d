// Exact decision of the folded join's candidates: every candidate's
// similarity in FP64 from the caller's CSR, kept if >= t.
//
// A warp takes up to 32 consecutive candidates: their row numbers and row
// pointers load one candidate per lane, then the warp computes them in turn
// (warp_dot). The sum's order differs from the oracle's ascending feature order, so a sum
// within the FP64 rounding of t is redone in that order by one lane; every
// decision is then the oracle's. The order depends on the two rows alone, so
// a pair's value does not depend on how the join was cut.
//
// Bound: instructions of the merge (n = 60k, d = 50k, t = 0.5 in FP32: 3.2M
// candidates in 1.63 ms, 427 warp instructions each, 73% of the issue slots
// at 32 warps a SM; more warps in fewer registers, votes in place of the
// shuffles of the chunks' ends and sums of four candidates at a time change
// nothing). Rows come from L2, which is at 12%.
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

// Warp dot product of rows S (shorter) and L: lane l sums the products of
// S's entries l, l + 32, ... in ascending order, the lanes' sums are added in
// a fixed tree.
//
// Rows of similar length are merged in chunks of 32 entries held in
// registers: every lane finds its S entry among the 32 L entries by shuffles,
// then the chunk that ends first moves on (its successor is already loaded).
// A much longer L is searched in place instead, kSearch entries of S a lane
// at a time so that the searches' loads overlap.
constexpr int kSearch = 4;
constexpr int kSearchRatio = 12;  // L at least this many times longer: searched

__device__ __forceinline__ double warp_dot(const int32_t* __restrict__ cs,
                                           const float* __restrict__ vs, int sl,
                                           const int32_t* __restrict__ cl,
                                           const float* __restrict__ vl, int ll, int lane) {
  double s = 0.0;
  if (ll >= kSearchRatio * sl) {
    for (int e0 = lane; e0 < sl; e0 += 32 * kSearch) {
      int32_t c[kSearch];
      int x[kSearch];
#pragma unroll
      for (int q = 0; q < kSearch; ++q) {
        c[q] = e0 + 32 * q < sl ? cs[e0 + 32 * q] : INT32_MAX;
        x[q] = 0;
      }
      for (int n = ll; n > 0;) {  // lower bounds of c in cl: each in [x, x + n]
        const int h = (n + 1) >> 1;
#pragma unroll
        for (int q = 0; q < kSearch; ++q)
          if (cl[x[q] + h - 1] < c[q]) x[q] += h;
        n -= h;
      }
#pragma unroll
      for (int q = 0; q < kSearch; ++q)
        if (e0 + 32 * q < sl && x[q] < ll && cl[x[q]] == c[q])
          s += (double)vs[e0 + 32 * q] * (double)vl[x[q]];
    }
  } else {
    int i = 32, j = 32;  // next chunk of S and L
    int32_t a = lane < sl ? cs[lane] : INT32_MAX, b = lane < ll ? cl[lane] : INT32_MAX;
    float av = lane < sl ? vs[lane] : 0.0f, bv = lane < ll ? vl[lane] : 0.0f;
    int32_t a2 = i + lane < sl ? cs[i + lane] : INT32_MAX;
    int32_t b2 = j + lane < ll ? cl[j + lane] : INT32_MAX;
    float av2 = i + lane < sl ? vs[i + lane] : 0.0f, bv2 = j + lane < ll ? vl[j + lane] : 0.0f;
    for (;;) {
      int p = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(kFull, b, p + o - 1) < a) p += o;
      const int32_t y = __shfl_sync(kFull, b, p);
      const float w = __shfl_sync(kFull, bv, p);
      if (y == a && a != INT32_MAX) s += (double)av * (double)w;
      const int32_t amax = __shfl_sync(kFull, a, 31), bmax = __shfl_sync(kFull, b, 31);
      if (amax <= bmax) {
        if (i >= sl) break;
        a = a2;
        av = av2;
        i += 32;
        a2 = i + lane < sl ? cs[i + lane] : INT32_MAX;
        av2 = i + lane < sl ? vs[i + lane] : 0.0f;
      }
      if (bmax <= amax) {
        if (j >= ll) break;
        b = b2;
        bv = bv2;
        j += 32;
        b2 = j + lane < ll ? cl[j + lane] : INT32_MAX;
        bv2 = j + lane < ll ? vl[j + lane] : 0.0f;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
  return s;
}

__global__ void __launch_bounds__(kThreads) k_verify(const VerifyArgs A) {
  const int64_t nc = (int64_t)*A.ncand;
  if (nc > A.cap) return;  // incomplete list: the host runs again with room
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  // candidates a warp takes at a time, from a counter: rows differ in length
  // by orders of magnitude
  int g = 32;
  while (g > 1 && (int64_t)g * 4 * warps > nc) g >>= 1;
  for (;;) {
    unsigned grp = 0;
    if (lane == 0) grp = atomicAdd(A.work, 1u);
    const int64_t base = (int64_t)__shfl_sync(kFull, grp, 0) * g;
    if (base >= nc) break;
    const int m = (int)(nc - base < g ? nc - base : g);
    uint32_t pi = 0, pj = 0;  // caller's rows
    uint32_t so = 0, lo = 0;  // first entry of the shorter and the longer row
    int sl = 0, ll = 0;       // their lengths
    bool swapped = false;     // the shorter row is J's
    double t = 0.0;
    if (lane < m) {
      const uint64_t key = A.cand[base + lane];
      const uint32_t ip = (uint32_t)(key >> 32), jp = (uint32_t)key;
      pi = A.permI ? (uint32_t)A.permI[ip] : ip;
      pj = A.permJ ? (uint32_t)A.permJ[jp] : jp;
      t = A.t_of_i ? (double)A.t_of_i[pi] : A.t_row ? (double)A.t_row[jp] : (double)A.t;
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
      const double s = warp_dot((sw_k ? A.colJ : A.colI) + so_k, (sw_k ? A.valJ : A.valI) + so_k,
                                sl_k, (sw_k ? A.colI : A.colJ) + lo_k,
                                (sw_k ? A.valI : A.valJ) + lo_k, ll_k, lane);
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
      uint64_t x = pi, y = (uint64_t)pj + (uint64_t)A.j_offset;
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
