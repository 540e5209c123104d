// Folded-bound tile kernel of the plain FP32 path: FP32 folded rows
// multiplied with FP32 FMA chains on the CUDA cores; pairs whose product
// reaches t - eps are listed (see fold.cuh).
//
// A tile is 128 I rows x 128 J rows. Two persistent CTAs a SM, each of eight
// compute warps (8 x 8 pairs a thread, as packed FMAs over column pairs) and
// a producer warp that copies 8 KB slices (16 columns x 128 rows) into two
// rings: I slices, which stay for a whole unit up to K = 128, and J slices.
// While one CTA's warps compare and list, the other's multiply.
//
// Bound: the FP32 FMA rate, 65 ns per column and tile on one SM (128 FMAs a
// clock); measured 92 ns per column and 0.38 us per tile at n = 60,000.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "fold_tile.cuh"

namespace cuapss {

namespace {

constexpr int kCW = 8;                                  // compute warps
constexpr int kThreads = 32 * (kCW + 1);                // + producer warp
constexpr int kI = kFoldResident32 / kFoldChunk32;      // I ring slots
constexpr int kJ = 5;                                   // J ring slots
constexpr int kRing = 4;                                // unit ids published ahead
constexpr int kHits = 48;                               // candidates a warp holds back
constexpr size_t kOffJ = (size_t)kI * kFoldSliceBytes;
constexpr size_t kOffHits = kOffJ + (size_t)kJ * kFoldSliceBytes;
constexpr size_t kOffBar = kOffHits + (size_t)kCW * kHits * 8;
constexpr int kBars = 2 * kI + 2 * kJ + 2 * kRing;
constexpr size_t kOffUnit = kOffBar + (size_t)kBars * 8;
constexpr size_t kSmem = kOffUnit + (size_t)kRing * 4 + 16;
static_assert(2 * (kSmem + 1024) <= 233472, "two CTAs a SM");

// Packed FP32 pairs.
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t twice(float x) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
  return d;
}
__device__ __forceinline__ float part(uint64_t v, int k) {
  return __uint_as_float((uint32_t)(k ? v >> 32 : v));
}

template <bool COUNT>
__global__ void __launch_bounds__(kThreads, 2) k_tiles_fold32(const __grid_constant__ FoldTileArgs A) {
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* ifull = reinterpret_cast<uint64_t*>(smem + kOffBar);
  uint64_t* iempty = ifull + kI;
  uint64_t* jfull = iempty + kI;
  uint64_t* jempty = jfull + kJ;
  uint64_t* ufull = jempty + kJ;
  uint64_t* uempty = ufull + kRing;
  volatile int* uring = reinterpret_cast<volatile int*>(smem + kOffUnit);
  volatile int* abort = reinterpret_cast<volatile int*>(smem + kOffUnit + kRing * 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kI; ++s) {
      mbar_init(&ifull[s], 1);
      mbar_init(&iempty[s], kCW);
    }
    for (int s = 0; s < kJ; ++s) {
      mbar_init(&jfull[s], 1);
      mbar_init(&jempty[s], kCW);
    }
    for (int k = 0; k < kRing; ++k) {
      mbar_init(&ufull[k], 1);
      mbar_init(&uempty[k], kCW);
    }
    *abort = 0;
    fence_mbar_init();
  }
  __syncthreads();
  allow_dependent_launch();

  if (warp == kCW) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t ii = 0, ij = 0;  // slices copied into each ring
      bool ok = true;
      for (uint32_t k = 0; ok; ++k) {
        const uint32_t slot = k % kRing, ur = k / kRing;
        if (!wait_abort(&uempty[slot], (ur & 1u) ^ 1u, abort)) {
          give_up(A.err, abort);
          break;
        }
        const int u = next_unit(A);
        uring[slot] = u;
        mbar_arrive(&ufull[slot]);
        if (u >= A.nunits) break;
        const FoldUnit U(A.units[u]);
        const FoldLevel& L = A.lev[U.lev];
        const int nkc = L.nkc;
        const uint8_t* srcI = L.I + (size_t)(U.I - L.firstI) * nkc * kFoldSliceBytes;
        for (int j = 0; ok && j < U.len; ++j) {
          const bool loadI = j == 0 || nkc > kI;
          const uint8_t* srcJ = L.J + (size_t)(U.J(j) - L.firstJ) * nkc * kFoldSliceBytes;
          for (int kc = 0; kc < nkc; ++kc) {
            if (loadI) {
              const uint32_t s = ii % kI, r = ii / kI;
              if (!wait_abort(&iempty[s], (r & 1u) ^ 1u, abort)) {
                give_up(A.err, abort);
                ok = false;
                break;
              }
              mbar_arrive_expect_tx(&ifull[s], kFoldSliceBytes);
              bulk_g2s(smem + (size_t)s * kFoldSliceBytes, srcI + (size_t)kc * kFoldSliceBytes,
                       kFoldSliceBytes, &ifull[s]);
              ++ii;
            }
            const uint32_t s = ij % kJ, r = ij / kJ;
            if (!wait_abort(&jempty[s], (r & 1u) ^ 1u, abort)) {
              give_up(A.err, abort);
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&jfull[s], kFoldSliceBytes);
            bulk_g2s(smem + kOffJ + (size_t)s * kFoldSliceBytes,
                     srcJ + (size_t)kc * kFoldSliceBytes, kFoldSliceBytes, &jfull[s]);
            ++ij;
          }
        }
      }
      // the last copies issued must have landed before the CTA exits
      for (uint32_t q = ii > kI ? ii - kI : 0u; q < ii; ++q)
        if (!mbar_wait(&ifull[q % kI], (q / kI) & 1u)) give_up(A.err, abort);
      for (uint32_t q = ij > kJ ? ij - kJ : 0u; q < ij; ++q)
        if (!mbar_wait(&jfull[q % kJ], (q / kJ) & 1u)) give_up(A.err, abort);
    }
    return;
  }
  // -------------------------------------------------------------- compute
  // thread (ty, tx): I rows 4 ty .. + 3 and 64 + 4 ty .. + 3, J rows likewise
  // with tx
  const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
  uint64_t* hits = reinterpret_cast<uint64_t*>(smem + kOffHits) + warp * kHits;
  int held = 0;  // candidates in hits, the same in every lane
  bool live = true, given_up = false;
  uint32_t ii = 0, ij = 0;  // first I slice of the unit or tile, J slices used
  for (uint32_t k = 0;; ++k) {
    const uint32_t slot = k % kRing, ur = k / kRing;
    live = warp_wait(&ufull[slot], ur & 1u, abort, A.err, live);
    const int u = live ? uring[slot] : A.nunits;
    __syncwarp();
    if (live && lane == 0) mbar_arrive(&uempty[slot]);
    if (u >= A.nunits) break;
    const FoldUnit U(A.units[u]);
    const int nkc = A.lev[U.lev].nkc;
    const float eps = A.lev[U.lev].eps;
    const bool stream = nkc > kI;
    const int64_t irow0 = (int64_t)U.I * kBlockRows;
    const int irows = (int)(A.nI - irow0 < kBlockRows ? A.nI - irow0 : kBlockRows);
    for (int jt = 0; jt < U.len; ++jt) {
      const int64_t jrow0 = (int64_t)U.J(jt) * kBlockRows;
      const int jrows = (int)(A.nJ - jrow0 < kBlockRows ? A.nJ - jrow0 : kBlockRows);
      const bool first = jt == 0, last = jt + 1 == U.len;
      uint64_t h[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) h[i][j] = 0ull;
      for (int kc = 0; kc < nkc; ++kc, ++ij) {
        const uint32_t qi = ii + (uint32_t)kc, si = qi % kI, sj = ij % kJ;
        if (first || stream) live = warp_wait(&ifull[si], (qi / kI) & 1u, abort, A.err, live);
        live = warp_wait(&jfull[sj], (ij / kJ) & 1u, abort, A.err, live);
        if (!live) break;
        const float4* a4 = reinterpret_cast<const float4*>(smem + (size_t)si * kFoldSliceBytes);
        const ulonglong2* b4 =
            reinterpret_cast<const ulonglong2*>(smem + kOffJ + (size_t)sj * kFoldSliceBytes);
#pragma unroll 4
        for (int c = 0; c < kFoldChunk32; ++c) {
          const float4 a0 = a4[c * 32 + ty], a1 = a4[c * 32 + 16 + ty];
          const ulonglong2 b0 = b4[c * 32 + tx], b1 = b4[c * 32 + 16 + tx];
          const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          const uint64_t bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t a = twice(av[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) h[i][j] = ffma2(a, bv[j], h[i][j]);
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&jempty[sj]);
          if (last || stream) mbar_arrive(&iempty[si]);
        }
      }
      if (stream || last) ii += (uint32_t)nkc;
      // ---- pairs at or above t - eps
      uint64_t pass = 0ull;  // bit 8 i + j
      if (live && !given_up) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = (j < 4 ? 0 : 64) + 4 * tx + (j & 3);
          float thr = A.t;
          if (A.t_row) thr = c < jrows ? A.t_row[jrow0 + c] : __int_as_float(0x7f800000);
          thr = __fsub_rd(thr, eps);
#pragma unroll
          for (int i = 0; i < 8; ++i)
            pass |= (uint64_t)(part(h[i][j >> 1], j & 1) >= thr) << (8 * i + j);
        }
      }
      if (__any_sync(0xffffffffu, pass != 0ull)) {
        // rows that exist, and in a self-join I rows below the J row
        for (uint64_t rest = pass; rest;) {
          const int b = __ffsll((long long)rest) - 1;
          rest &= rest - 1;
          const int i = b >> 3, j = b & 7;
          const int r = (i < 4 ? 0 : 64) + 4 * ty + (i & 3);
          const int c = (j < 4 ? 0 : 64) + 4 * tx + (j & 3);
          if (r >= irows || c >= jrows || (A.self && irow0 + r >= jrow0 + c))
            pass &= ~(1ull << b);
        }
        if (COUNT) {
          const uint32_t total = __reduce_add_sync(0xffffffffu, (uint32_t)__popcll(pass));
          if (lane == 0 && total)
            atomicAdd(&A.class_count[((size_t)U.lev * A.nbI + U.I) * A.nbJ + U.J(jt)], total);
        } else {
          for (;;) {  // one candidate of each thread that has some left
            const unsigned some = __ballot_sync(0xffffffffu, pass != 0ull);
            if (!some) break;
            if (held > kHits - 32) {
              given_up = flush_hits(A, hits, held, lane);
              held = 0;
              if (given_up) break;
            }
            if (pass) {
              const int b = __ffsll((long long)pass) - 1;
              pass &= pass - 1;
              const int i = b >> 3, j = b & 7;
              const int r = (i < 4 ? 0 : 64) + 4 * ty + (i & 3);
              const int c = (j < 4 ? 0 : 64) + 4 * tx + (j & 3);
              hits[held + __popc(some & ((1u << lane) - 1u))] =
                  ((uint64_t)(irow0 + r) << 32) | (uint64_t)(jrow0 + c);
            }
            held += __popc(some);
          }
        }
      }
    }
  }
  if (!COUNT && held > 0) flush_hits(A, hits, held, lane);
}

cuapss_status tiles_fold32_init() {
  static std::mutex mu;
  static uint64_t done = 0;  // bit per device
  int dev = 0;
  CU_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && ((done >> dev) & 1ull)) return CUAPSS_OK;
  CU_TRY(cudaFuncSetAttribute(k_tiles_fold32<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kSmem));
  CU_TRY(cudaFuncSetAttribute(k_tiles_fold32<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kSmem));
  if (dev < 64) done |= 1ull << dev;
  return CUAPSS_OK;
}

}  // namespace

cuapss_status launch_tiles_fold32(const FoldTileArgs& a, int sms, cudaStream_t st, bool count) {
  ST_TRY(tiles_fold32_init());
  if (a.nunits <= 0) return CUAPSS_OK;
  const int grid = std::min(a.nunits, 2 * sms);
  if (count) k_tiles_fold32<true><<<grid, kThreads, kSmem, st>>>(a);
  else k_tiles_fold32<false><<<grid, kThreads, kSmem, st>>>(a);
  LAUNCH_CHECK();
  return CUAPSS_OK;
}

}  // namespace cuapss
