// Folded-bound tile kernel: the folded rows of fold.cuh multiplied tile by
// tile on the 5th-generation tensor cores (tcgen05, FP32 accumulators in
// tensor memory); pairs whose product reaches t - eps are listed.
//
// A tile is 256 I rows (two row blocks, the N side) x 128 J rows (the M
// side, one tensor-memory lane each). Warp roles, one persistent CTA per SM:
//   warp 0     producer: bulk copies of pre-swizzled 16 KB chunks (128 rows x
//              64 columns) into two rings, A (J chunks, kA slots of 16 KB)
//              and B (I chunk pairs, kB slots of 32 KB);
//   warp 1     MMA: one thread issues M = 128, N = 256, K = 16 MMAs into two
//              alternating accumulators of 256 columns (all of tensor memory);
//   warps 2-9  epilogue, two per lane quarter (one I block each): the largest
//              of each J row's 128 products is compared with t - eps; only
//              32-column groups in which some row reaches it are read again
//              and listed.
// Up to kB chunks wide (K <= 256), the I chunks stay in the B ring for a
// whole unit (I pair x range of J blocks) and only 16 KB per 64 columns move
// from L2 per tile, a third of what streaming both operands takes; wider
// folds stream both.
//
// Bound: the tensor cores (K / 64 x 512 cycles per tile) down to K = 128; at
// K = 64 the epilogue's 256 tensor-memory columns per lane quarter cost
// about as much as the MMAs.
//
// Every wait is bounded as in tile_mma.cu: a timeout raises kErrTimeout and
// a shared abort flag, copies and MMAs in flight are drained, tensor memory
// is freed and the kernel returns.
#include <cuda_runtime.h>

#include <mutex>

#include "fold.cuh"
#include "ptx.cuh"

namespace cuapss {

namespace {

constexpr int kA = 6;                     // A ring slots (16 KB)
constexpr int kB = 4;                     // B ring slots (32 KB)
constexpr int kEW = 8;                    // epilogue warps
constexpr int kThreads = 64 + 32 * kEW;
constexpr int kRing = 4;                  // unit ids published ahead
constexpr int kReaders = 1 + kEW;         // MMA thread + epilogue warps
constexpr int kColsPerAcc = 256;
constexpr int kBars = 2 * kA + 2 * kB + 4 + 2 * kRing + 1;
constexpr size_t kOffB = (size_t)kA * kFoldTileBytes;
constexpr size_t kOffBar = kOffB + (size_t)kB * 2 * kFoldTileBytes;
constexpr size_t kOffUnit = kOffBar + (size_t)kBars * 8;
constexpr size_t kOffMisc = kOffUnit + (size_t)kRing * 16 + 8;
constexpr size_t kSmem = kOffMisc + 16 + 1024;  // + alignment slack
static_assert(kSmem <= 232448, "shared memory budget");
static_assert(kOffUnit % 8 == 0, "unit ring alignment");

__device__ __forceinline__ bool wait_abort(uint64_t* bar, uint32_t parity,
                                           const volatile int* abort) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t i = 0; i < kMaxPolls; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort || globaltimer_ns() - t0 >= kWaitLimitNs) return false;
  }
  return false;
}

__device__ __forceinline__ void give_up(int* err, volatile int* abort) {
  if (!*abort) {
    *abort = 1;
    atomicOr(err, kErrTimeout);
  }
}

__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort,
                                          int* err, bool live) {
  bool got = live ? wait_abort(bar, parity, abort) : true;
  got = __all_sync(0xffffffffu, got);
  if (live && !got && (threadIdx.x & 31) == 0) give_up(err, abort);
  return live && got;
}

struct Unit {
  int I, J0, J1, lev;
};

template <bool COUNT>
__global__ void __launch_bounds__(kThreads, 1) k_tiles_fold(const __grid_constant__ FoldTileArgs A) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<size_t>(smem_raw) + 1023) & ~(size_t)1023);
  uint8_t* ringA = base;
  uint8_t* ringB = base + kOffB;
  uint64_t* afull = reinterpret_cast<uint64_t*>(base + kOffBar);
  uint64_t* aempty = afull + kA;
  uint64_t* bfull = aempty + kA;
  uint64_t* bempty = bfull + kB;
  uint64_t* tfull = bempty + kB;
  uint64_t* tempty = tfull + 2;
  uint64_t* ufull = tempty + 2;
  uint64_t* uempty = ufull + kRing;
  uint64_t* drain = uempty + kRing;
  volatile int* uring = reinterpret_cast<volatile int*>(base + kOffUnit);
  uint32_t* tmem_base = reinterpret_cast<uint32_t*>(base + kOffMisc);
  volatile int* abort = reinterpret_cast<volatile int*>(base + kOffMisc + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kA; ++s) {
      mbar_init(&afull[s], 1);
      mbar_init(&aempty[s], 1);
    }
    for (int s = 0; s < kB; ++s) {
      mbar_init(&bfull[s], 1);
      mbar_init(&bempty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], kEW);
    }
    for (int k = 0; k < kRing; ++k) {
      mbar_init(&ufull[k], 1);
      mbar_init(&uempty[k], kReaders);
    }
    mbar_init(drain, 1);
    *abort = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base;
  allow_dependent_launch();

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      uint32_t ia = 0, ib = 0;  // chunks copied into each ring
      bool ok = true;
      for (uint32_t k = 0; ok; ++k) {
        const uint32_t slot = k % kRing, ur = k / kRing;
        if (!wait_abort(&uempty[slot], (ur & 1u) ^ 1u, abort)) {
          give_up(A.err, abort);
          break;
        }
        const int u = atomicAdd(A.unit_counter, 1);
        uring[slot] = u;
        mbar_arrive(&ufull[slot]);
        if (u >= A.nunits) break;
        const int4 U = A.units[u];
        const FoldLevel& L = A.lev[U.w];
        const int nkc = L.nkc;
        const int wI = U.x + 1 < A.nbI ? 2 : 1;
        const uint8_t* srcI = L.I + (size_t)(U.x - L.firstI) * nkc * kFoldTileBytes;
        const uint8_t* srcJ = L.J + (size_t)(U.y - L.firstJ) * nkc * kFoldTileBytes;
        for (int J = U.y; ok && J < U.z; ++J) {
          const bool loadB = J == U.y || nkc > kB;
          for (int kc = 0; kc < nkc; ++kc) {
            if (loadB) {
              const uint32_t s = ib % kB, r = ib / kB;
              if (!wait_abort(&bempty[s], (r & 1u) ^ 1u, abort)) {
                give_up(A.err, abort);
                ok = false;
                break;
              }
              uint8_t* dst = ringB + (size_t)s * 2 * kFoldTileBytes;
              mbar_arrive_expect_tx(&bfull[s], (uint32_t)wI * kFoldTileBytes);
              bulk_g2s(dst, srcI + (size_t)kc * kFoldTileBytes, kFoldTileBytes, &bfull[s]);
              if (wI == 2)
                bulk_g2s(dst + kFoldTileBytes, srcI + (size_t)(nkc + kc) * kFoldTileBytes,
                         kFoldTileBytes, &bfull[s]);
              ++ib;
            }
            const uint32_t s = ia % kA, r = ia / kA;
            if (!wait_abort(&aempty[s], (r & 1u) ^ 1u, abort)) {
              give_up(A.err, abort);
              ok = false;
              break;
            }
            mbar_arrive_expect_tx(&afull[s], kFoldTileBytes);
            bulk_g2s(ringA + (size_t)s * kFoldTileBytes, srcJ, kFoldTileBytes, &afull[s]);
            srcJ += kFoldTileBytes;
            ++ia;
          }
        }
      }
      // the last copies issued must have landed before the CTA exits
      for (uint32_t q = ia > kA ? ia - kA : 0u; q < ia; ++q)
        if (!mbar_wait(&afull[q % kA], (q / kA) & 1u)) give_up(A.err, abort);
      for (uint32_t q = ib > kB ? ib - kB : 0u; q < ib; ++q)
        if (!mbar_wait(&bfull[q % kB], (q / kB) & 1u)) give_up(A.err, abort);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ----------------------------------------------------------------- MMA
    if (lane == 0) {
      const uint32_t idesc1 = umma_idesc_bf16(kBlockRows, kBlockRows);
      const uint32_t idesc2 = umma_idesc_bf16(kBlockRows, 2 * kBlockRows);
      uint32_t ia = 0, ib = 0, tt = 0;  // A chunks used, first B chunk of the unit or tile, tiles
      bool ok = true;
      for (uint32_t k = 0; ok; ++k) {
        const uint32_t slot = k % kRing, ur = k / kRing;
        if (!wait_abort(&ufull[slot], ur & 1u, abort)) {
          give_up(A.err, abort);
          break;
        }
        const int u = uring[slot];
        mbar_arrive(&uempty[slot]);
        if (u >= A.nunits) break;
        const int4 U = A.units[u];
        const int nkc = A.lev[U.w].nkc;
        const bool stream = nkc > kB;
        const uint32_t idesc = U.x + 1 < A.nbI ? idesc2 : idesc1;
        for (int J = U.y; ok && J < U.z; ++J, ++tt) {
          const bool first = J == U.y, last = J + 1 == U.z;
          const uint32_t b = tt & 1u, tr = tt >> 1;
          if (!wait_abort(&tempty[b], (tr & 1u) ^ 1u, abort)) {
            give_up(A.err, abort);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + b * (uint32_t)kColsPerAcc;
          for (int kc = 0; kc < nkc; ++kc, ++ia) {
            const uint32_t qb = ib + (uint32_t)kc;
            if ((first || stream) && !wait_abort(&bfull[qb % kB], (qb / kB) & 1u, abort)) {
              give_up(A.err, abort);
              ok = false;
              break;
            }
            const uint32_t s = ia % kA;
            if (!wait_abort(&afull[s], (ia / kA) & 1u, abort)) {
              give_up(A.err, abort);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t ad = umma_desc_sw128(ringA + (size_t)s * kFoldTileBytes);
            const uint64_t bd = umma_desc_sw128(ringB + (size_t)(qb % kB) * 2 * kFoldTileBytes);
#pragma unroll
            for (int q = 0; q < 4; ++q)
              umma_bf16(d, ad + 2u * q, bd + 2u * q, idesc, (kc | q) != 0 ? 1u : 0u);
            umma_commit(&aempty[s]);
            if (last || stream) umma_commit(&bempty[qb % kB]);
          }
          if (ok) umma_commit(&tfull[b]);
          if (stream || last) ib += (uint32_t)nkc;
        }
      }
      // every MMA issued must be complete before tensor memory is freed
      if (ia > 0) {
        umma_commit(drain);
        if (!mbar_wait(drain, 0)) give_up(A.err, abort);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------- epilogue
    const int q4 = warp & 3;             // tensor-memory lane quarter of this warp
    const int half = (warp - 2) >> 2;    // which of the two I blocks
    const int row = 32 * q4 + lane;      // J row within its block
    bool live = true;
    uint32_t tt = 0;
    for (uint32_t k = 0;; ++k) {
      const uint32_t slot = k % kRing, ur = k / kRing;
      live = warp_wait(&ufull[slot], ur & 1u, abort, A.err, live);
      const int u = live ? uring[slot] : A.nunits;
      __syncwarp();
      if (live && lane == 0) mbar_arrive(&uempty[slot]);
      if (u >= A.nunits) break;
      const int4 U = A.units[u];
      const float eps = A.lev[U.w].eps;
      const int I = U.x + half;
      const bool haveI = I < A.nbI;
      const int64_t irow0 = (int64_t)I * kBlockRows;
      const int icols = haveI ? (int)(A.nI - irow0 < kBlockRows ? A.nI - irow0 : kBlockRows) : 0;
      for (int J = U.y; J < U.z; ++J, ++tt) {
        const uint32_t b = tt & 1u, tr = tt >> 1;
        const int64_t jrow = (int64_t)J * kBlockRows + row;
        const float thr =
            jrow < A.nJ ? __fsub_rd(A.t_row ? A.t_row[jrow] : A.t, eps) : __int_as_float(0x7f800000);
        live = warp_wait(&tfull[b], tr & 1u, abort, A.err, live);
        tc_fence_after();
        const uint32_t taddr = tmem + b * (uint32_t)kColsPerAcc + (uint32_t)(half * kBlockRows) +
                               ((uint32_t)(32 * q4) << 16);
        if (live && haveI && !(A.self && J < I)) {
          uint32_t hit = 0;  // bit g: some product of columns 32 g .. reaches thr
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t v[32];
            tmem_ld32(taddr + 32u * g, v);
            float m = __uint_as_float(v[0]);
#pragma unroll
            for (int j = 1; j < 32; ++j) m = fmaxf(m, __uint_as_float(v[j]));
            hit |= (uint32_t)(m >= thr) << g;
          }
          const uint32_t any = __reduce_or_sync(0xffffffffu, hit);
          if (any) {
            uint32_t n_hits = 0;
            const int64_t jmin = A.self ? jrow : INT64_MAX;  // self: I rows below the J row only
            for (int g = 0; g < 4; ++g) {
              if (!((any >> g) & 1u)) continue;  // warp-uniform
              uint32_t v[32];
              tmem_ld32(taddr + 32u * g, v);
              uint32_t pass = 0;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                pass |= (uint32_t)(__uint_as_float(v[j]) >= thr) << j;
              // columns that exist, and for a self-join lie below the J row
              int64_t lim = jmin - irow0 < (int64_t)icols ? jmin - irow0 : (int64_t)icols;
              const int c = (int)lim - 32 * g;
              pass &= c >= 32 ? 0xffffffffu : c <= 0 ? 0u : (1u << c) - 1u;
              const int mine = __popc(pass);
              if (COUNT) {
                n_hits += (uint32_t)mine;
              } else if (__any_sync(0xffffffffu, mine != 0)) {
                int incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                  const int x = __shfl_up_sync(0xffffffffu, incl, o);
                  if (lane >= o) incl += x;
                }
                unsigned long long w = 0;
                if (lane == 31) w = atomicAdd(A.cand_count, (unsigned long long)incl);
                w = __shfl_sync(0xffffffffu, w, 31) + (unsigned long long)(incl - mine);
                while (pass) {
                  const int j = __ffs(pass) - 1;
                  pass &= pass - 1;
                  if ((int64_t)w < A.cand_cap)
                    A.cand[w] = ((uint64_t)(irow0 + 32 * g + j) << 32) | (uint64_t)jrow;
                  ++w;
                }
              }
            }
            if (COUNT) {
              const uint32_t total = __reduce_add_sync(0xffffffffu, n_hits);
              if (lane == 0 && total)
                atomicAdd(&A.class_count[((size_t)U.w * A.nbI + I) * A.nbJ + J], total);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (live && lane == 0) mbar_arrive(&tempty[b]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

cuapss_status tiles_fold_init() {
  static std::mutex mu;
  static uint64_t done = 0;  // bit per device
  int dev = 0;
  CU_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && ((done >> dev) & 1ull)) return CUAPSS_OK;
  CU_TRY(cudaFuncSetAttribute(k_tiles_fold<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kSmem));
  CU_TRY(cudaFuncSetAttribute(k_tiles_fold<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kSmem));
  if (dev < 64) done |= 1ull << dev;
  return CUAPSS_OK;
}

}  // namespace

cuapss_status launch_tiles_fold(const FoldTileArgs& a, int grid, cudaStream_t st, bool count) {
  ST_TRY(tiles_fold_init());
  if (a.nunits <= 0) return CUAPSS_OK;
  if (count) k_tiles_fold<true><<<grid, kThreads, kSmem, st>>>(a);
  else k_tiles_fold<false><<<grid, kThreads, kSmem, st>>>(a);
  LAUNCH_CHECK();
  return CUAPSS_OK;
}

}  // namespace cuapss
