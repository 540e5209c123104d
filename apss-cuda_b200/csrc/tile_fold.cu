// Folded-bound tile kernel: the folded rows of fold.cuh multiplied tile by
// tile on the 5th-generation tensor cores (tcgen05, FP32 accumulators in
// tensor memory); pairs whose product reaches t - eps are listed.
//
// A tile is 256 I rows (two row blocks, the N side) x 128 J rows (the M
// side, one tensor-memory lane each). Warp roles, one persistent CTA per SM:
//   warp 0     producer: bulk copies of pre-swizzled 16 KB chunks (128 rows x
//              64 columns) into two rings, A (J chunks, kA slots of 16 KB)
//              and B (I chunk pairs, kB slots of 32 KB);
//   warps 1-2  MMA: each issues the M = 128, N = 256, K = 16 MMAs of every
//              other tile into its own accumulator of 256 columns (the two
//              are all of tensor memory);
//   warps 4-11 epilogue, two per lane quarter (one I block each): a warp
//              loads its 128 columns, gives the accumulator back, and votes
//              once on the largest of each J row's products against t - eps;
//              only where that passes are the column groups looked at one by
//              one. Candidates gather in shared memory, so that a warp
//              reserves list room once per about 100 of them (one
//              reservation per group cost a global atomic's latency each:
//              n = 400,000, 3 candidates a tile, 29 ms).
// Up to kB chunks wide (K <= 256), the I chunks stay in the B ring for a
// whole unit (I pair x range of J blocks) and only 16 KB per 64 columns move
// from L2 per tile, a third of what streaming both operands takes; wider
// folds stream both.
//
// Bound: the tensor cores from K = 128 on (260 ns per 64 columns and tile at
// their peak; measured 709 ns at K = 128, 1,371 at 256, of which the loads and
// hand-offs hide all but 60); at K = 64 (613 ns) the hand-off of the two
// accumulators: tensor cores, epilogue loads and waits in turn, tensor pipe
// 51% active; above K = 256 the operand stream from L2 (about 410 ns per 64
// columns). Holding the accumulator until a warp was done, voting per column
// group: 616, 873 and 1,446 ns at K = 64, 128 and 256. Sixteen epilogue warps
// of 64 columns each: 630, 825, 1,453 (more warps wait and poll, the loads are
// no faster).
//
// Every wait is bounded as in tile_mma.cu: a timeout raises kErrTimeout and
// a shared abort flag, copies and MMAs in flight are drained, tensor memory
// is freed and the kernel returns.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "fold.cuh"
#include "fold_tile.cuh"
#include "ptx.cuh"

namespace cuapss {

namespace {

constexpr int kA = 5;                     // A ring slots (16 KB)
constexpr int kB = kFoldResident16 / kFoldChunk16;   // B ring slots (32 KB)
constexpr int kMW = 2;                    // MMA warps, one per accumulator
constexpr int kEW = 8;                    // epilogue warps
constexpr int kEpiCols = 1024 / kEW;      // accumulator columns of an epilogue warp
constexpr int kFirstEpi = 4;              // a multiple of 4: lane quarter = warp % 4
constexpr int kThreads = 32 * (kFirstEpi + kEW);
constexpr int kRing = 4;                  // unit ids published ahead
constexpr int kReaders = kMW + kEW;       // MMA and epilogue warps
constexpr int kColsPerAcc = 256;
constexpr int kBars = (kMW + 1) * kA + 2 * kB + 4 + 2 * kRing + kMW;
constexpr size_t kOffB = (size_t)kA * kFoldTileBytes;
constexpr int kHits = 1024 / kEW;               // candidates an epilogue warp holds back
constexpr size_t kOffHits = kOffB + (size_t)kB * 2 * kFoldTileBytes;
constexpr size_t kOffBar = kOffHits + (size_t)kEW * kHits * 8;
constexpr size_t kOffUnit = kOffBar + (size_t)kBars * 8;
constexpr size_t kOffMisc = kOffUnit + (size_t)kRing * 16 + 8;
constexpr size_t kSmem = kOffMisc + 16 + 1024;  // + alignment slack
static_assert(kSmem <= 232448, "shared memory budget");
static_assert(kOffUnit % 8 == 0, "unit ring alignment");

// One 32-column group of a J row's products: the columns at or above thr
// (bit j of the result), c of which exist (and, in a self-join, lie below
// the J row).
__device__ __forceinline__ uint32_t passing(const uint32_t (&v)[32], float thr, int c) {
  uint32_t pass = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) pass |= (uint32_t)(__uint_as_float(v[j]) >= thr) << j;
  return pass & (c >= 32 ? 0xffffffffu : c <= 0 ? 0u : (1u << c) - 1u);
}

__device__ __forceinline__ float max3(float a, uint32_t b, uint32_t c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(__uint_as_float(b)), "f"(__uint_as_float(c)));
  return d;
}

// Three-input maxima: half the instructions of the epilogue's main loop.
__device__ __forceinline__ float largest(const uint32_t (&v)[32]) {
  float m[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) m[q] = __uint_as_float(v[q]);
#pragma unroll
  for (int j = 2; j + 1 < 32; j += 2) m[(j >> 1) & 1] = max3(m[(j >> 1) & 1], v[j], v[j + 1]);
  return fmaxf(m[0], m[1]);
}

template <bool COUNT>
__global__ void __launch_bounds__(kThreads, 1) k_tiles_fold(const __grid_constant__ FoldTileArgs A) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<size_t>(smem_raw) + 1023) & ~(size_t)1023);
  uint8_t* ringA = base;
  uint8_t* ringB = base + kOffB;
  // afull[m kA + s]: slot s was filled for MMA warp m. A barrier per warp and
  // slot, so that a warp sees every phase of the barriers it waits on (a wait
  // on a phase's parity is only meaningful one phase ahead).
  uint64_t* afull = reinterpret_cast<uint64_t*>(base + kOffBar);
  uint64_t* aempty = afull + kMW * kA;
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
    for (int s = 0; s < kMW * kA; ++s) mbar_init(&afull[s], 1);
    for (int s = 0; s < kA; ++s) mbar_init(&aempty[s], 1);
    for (int s = 0; s < kB; ++s) {
      mbar_init(&bfull[s], 1);
      mbar_init(&bempty[s], kMW);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], kEW);
    }
    for (int k = 0; k < kRing; ++k) {
      mbar_init(&ufull[k], 1);
      mbar_init(&uempty[k], kReaders);
    }
    for (int m = 0; m < kMW; ++m) mbar_init(&drain[m], 1);
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
      uint32_t ia = 0, ib = 0, tt = 0;  // chunks copied into each ring, tiles
      uint32_t use[kMW] = {};           // bit s: parity of the next use of afull[m kA + s]
      uint32_t last_m = 0, last_p = 0;  // bit s: warp and parity of slot s's last use
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
        const int wI = U.I + 1 < A.nbI && !U.single ? 2 : 1;
        const uint8_t* srcI = L.I + (size_t)(U.I - L.firstI) * nkc * kFoldTileBytes;
        for (int j = 0; ok && j < U.len; ++j, ++tt) {
          const uint32_t m = tt & 1u;
          const bool loadB = j == 0 || nkc > kB;
          const uint8_t* srcJ = L.J + (size_t)(U.J(j) - L.firstJ) * nkc * kFoldTileBytes;
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
            mbar_arrive_expect_tx(&afull[m * kA + s], kFoldTileBytes);
            bulk_g2s(ringA + (size_t)s * kFoldTileBytes, srcJ, kFoldTileBytes, &afull[m * kA + s]);
            srcJ += kFoldTileBytes;
            const uint32_t bit = 1u << s, p = (m ? use[1] : use[0]) & bit;
            last_m = (last_m & ~bit) | (m << s);
            last_p = (last_p & ~bit) | p;
            if (m) use[1] ^= bit;
            else use[0] ^= bit;
            ++ia;
          }
        }
      }
      // the last copies issued must have landed before the CTA exits
      for (uint32_t s = 0; s < (ia < kA ? ia : (uint32_t)kA); ++s)
        if (!mbar_wait(&afull[((last_m >> s) & 1u) * kA + s], (last_p >> s) & 1u))
          give_up(A.err, abort);
      for (uint32_t q = ib > kB ? ib - kB : 0u; q < ib; ++q)
        if (!mbar_wait(&bfull[q % kB], (q / kB) & 1u)) give_up(A.err, abort);
    }
    __syncwarp();
  } else if (warp <= kMW) {
    // ----------------------------------------------------------------- MMA
    // MMA warp m takes tiles m, m + 2, ... (accumulator m): issuing a tile's
    // MMAs, waits and commits takes its warp about as long as the tensor
    // cores take to run them, so two warps keep the cores fed
    const uint32_t m = (uint32_t)warp - 1u;
    const uint32_t idesc1 = umma_idesc_bf16(kBlockRows, kBlockRows);
    const uint32_t idesc2 = umma_idesc_bf16(kBlockRows, 2 * kBlockRows);
    const uint64_t descA = umma_desc_sw128(ringA), descB = umma_desc_sw128(ringB);
    const uint32_t d = tmem + m * (uint32_t)kColsPerAcc;
    uint32_t ia = 0;          // A chunks before this tile
    uint32_t ib = 0, tt = 0;  // first B chunk of the unit or tile, tiles
    uint32_t use = 0;         // bit s: parity of the next use of afull[m kA + s]
    bool live = true;
    for (uint32_t k = 0;; ++k) {
      const uint32_t slot = k % kRing, ur = k / kRing;
      live = warp_wait(&ufull[slot], ur & 1u, abort, A.err, live);
      const int u = live ? uring[slot] : A.nunits;
      __syncwarp();
      if (live && lane == 0) mbar_arrive(&uempty[slot]);
      if (u >= A.nunits) break;
      const FoldUnit U(A.units[u]);
      const int nkc = A.lev[U.lev].nkc;
      const bool stream = nkc > kB;
      const uint32_t idesc = U.I + 1 < A.nbI && !U.single ? idesc2 : idesc1;
      bool fresh = true;  // this warp has not waited for the unit's B chunks
      for (int j = 0; live && j < U.len; ++j, ++tt, ia += (uint32_t)nkc) {
        if ((tt & 1u) == m) {
          // the warp's last tile of the unit releases the resident B chunks
          const bool last = j + kMW >= U.len;
          live = warp_wait(&tempty[m], ((tt >> 1) & 1u) ^ 1u, abort, A.err, live);
          tc_fence_after();
          for (int kc = 0; kc < nkc; ++kc) {
            const uint32_t qb = ib + (uint32_t)kc, sb = qb % kB, sa = (ia + (uint32_t)kc) % kA;
            if (fresh || stream)
              live = warp_wait(&bfull[sb], (qb / kB) & 1u, abort, A.err, live);
            live = warp_wait(&afull[m * kA + sa], (use >> sa) & 1u, abort, A.err, live);
            if (!live) break;
            use ^= 1u << sa;
            tc_fence_after();
            const uint64_t ad = descA + (uint64_t)(sa * (kFoldTileBytes >> 4));
            const uint64_t bd = descB + (uint64_t)(sb * (2 * kFoldTileBytes >> 4));
#pragma unroll
            for (int q = 0; q < 4; ++q)
              umma_bf16_warp(d, ad + 2u * q, bd + 2u * q, idesc, (kc | q) != 0 ? 1u : 0u);
            umma_commit_warp(&aempty[sa]);
            if (last || stream) umma_commit_warp(&bempty[sb]);
          }
          if (live) umma_commit_warp(&tfull[m]);
          fresh = false;
        } else if (stream) {
          // the other warp's tile: its B chunks are seen and released here too
          for (int kc = 0; kc < nkc; ++kc) {
            const uint32_t qb = ib + (uint32_t)kc, sb = qb % kB;
            live = warp_wait(&bfull[sb], (qb / kB) & 1u, abort, A.err, live);
            if (live && lane == 0) mbar_arrive(&bempty[sb]);
          }
        }
        if (stream) ib += (uint32_t)nkc;
      }
      if (!stream) {
        // a unit of one tile leaves the other warp without one: it sees and
        // releases the B chunks all the same
        if (fresh)
          for (int kc = 0; kc < nkc; ++kc) {
            const uint32_t qb = ib + (uint32_t)kc, sb = qb % kB;
            live = warp_wait(&bfull[sb], (qb / kB) & 1u, abort, A.err, live);
            if (live && lane == 0) mbar_arrive(&bempty[sb]);
          }
        ib += (uint32_t)nkc;
      }
    }
    // every MMA issued must be complete before tensor memory is freed
    umma_commit_warp(&drain[m]);
    if (!mbar_wait(&drain[m], 0) && lane == 0) give_up(A.err, abort);
    __syncwarp();
  } else if (warp >= kFirstEpi) {
    // ------------------------------------------------------------- epilogue
    const int q4 = warp & 3;             // tensor-memory lane quarter of this warp
    const int strip = (warp - kFirstEpi) >> 2;      // which kEpiCols columns
    const int half = strip * kEpiCols / kBlockRows; // which of the two I blocks
    const int col0 = strip * kEpiCols % kBlockRows; // first column within it
    const int row = 32 * q4 + lane;      // J row within its block
    uint64_t* hits = reinterpret_cast<uint64_t*>(base + kOffHits) + (warp - kFirstEpi) * kHits;
    int held = 0;                        // candidates in hits, the same in every lane
    bool live = true, given_up = false;
    uint32_t tt = 0;
    for (uint32_t k = 0;; ++k) {
      const uint32_t slot = k % kRing, ur = k / kRing;
      live = warp_wait(&ufull[slot], ur & 1u, abort, A.err, live);
      const int u = live ? uring[slot] : A.nunits;
      __syncwarp();
      if (live && lane == 0) mbar_arrive(&uempty[slot]);
      if (u >= A.nunits) break;
      const FoldUnit U(A.units[u]);
      const float eps = A.lev[U.lev].eps;
      const int I = U.I + half;
      const bool haveI = I < A.nbI && !(half == 1 && U.single);
      const int64_t irow0 = (int64_t)I * kBlockRows + col0;  // I row of this warp's first column
      const int icols =
          haveI && A.nI > irow0 ? (int)(A.nI - irow0 < kEpiCols ? A.nI - irow0 : kEpiCols) : 0;
      for (int j = 0; j < U.len; ++j, ++tt) {
        const int J = U.J(j);
        const uint32_t b = tt & 1u, tr = tt >> 1;
        const int64_t jrow = (int64_t)J * kBlockRows + row;
        const float thr =
            jrow < A.nJ ? __fsub_rd(A.t_row ? A.t_row[jrow] : A.t, eps) : __int_as_float(0x7f800000);
        live = warp_wait(&tfull[b], tr & 1u, abort, A.err, live);
        tc_fence_after();
        const uint32_t taddr = tmem + b * (uint32_t)kColsPerAcc + (uint32_t)(strip * kEpiCols) +
                               ((uint32_t)(32 * q4) << 16);
        const bool work = live && haveI && !(A.self && J < I);
        uint32_t v[kEpiCols / 32][32];
        if (work) {
#pragma unroll
          for (int g = 0; g < kEpiCols / 32; ++g) tmem_ld32_async(taddr + 32u * g, v[g]);
#pragma unroll
          for (int g = 0; g < kEpiCols / 32; ++g) tmem_wait(v[g]);
        }
        // the products are in registers: the accumulator is free again
        tc_fence_before();
        __syncwarp();
        if (live && lane == 0) mbar_arrive(&tempty[b]);
        if (!work || given_up) continue;
        // the groups' maxima first, and one vote: nearly all tiles end here
        float m[kEpiCols / 32];
        float top = largest(v[0]);
        m[0] = top;
#pragma unroll
        for (int g = 1; g < kEpiCols / 32; ++g) {
          m[g] = largest(v[g]);
          top = fmaxf(top, m[g]);
        }
        if (__any_sync(0xffffffffu, top >= thr)) {
          // columns that exist; for a self-join only those below the J row
          int64_t lim = icols;
          if (A.self && jrow - irow0 < lim) lim = jrow - irow0;
          uint32_t n_hits = 0;
#pragma unroll
          for (int g = 0; g < kEpiCols / 32; ++g) {
            if (given_up || !__any_sync(0xffffffffu, m[g] >= thr)) continue;
            uint32_t pass = passing(v[g], thr, (int)lim - 32 * g);
            if (COUNT) {
              n_hits += (uint32_t)__popc(pass);
              continue;
            }
            for (;;) {  // one candidate of each row that has some left
              const unsigned some = __ballot_sync(0xffffffffu, pass != 0u);
              if (!some) break;
              if (held > kHits - 32) {
                given_up = flush_hits(A, hits, held, lane);
                held = 0;
                if (given_up) break;
              }
              if (pass) {
                const int j = __ffs(pass) - 1;
                pass &= pass - 1;
                hits[held + __popc(some & ((1u << lane) - 1u))] =
                    ((uint64_t)(irow0 + 32 * g + j) << 32) | (uint64_t)jrow;
              }
              held += __popc(some);
            }
          }
          if (COUNT) {
            const uint32_t total = __reduce_add_sync(0xffffffffu, n_hits);
            if (lane == 0 && total)
              atomicAdd(&A.class_count[((size_t)U.lev * A.nbI + I) * A.nbJ + J], total);
          }
        }
      }
    }
    if (!COUNT && held > 0) flush_hits(A, hits, held, lane);
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

cuapss_status launch_tiles_fold(const FoldTileArgs& a, int sms, cudaStream_t st, bool count) {
  ST_TRY(tiles_fold_init());
  if (a.nunits <= 0) return CUAPSS_OK;
  const int grid = std::min(a.nunits, sms);
  if (count) k_tiles_fold<true><<<grid, kThreads, kSmem, st>>>(a);
  else k_tiles_fold<false><<<grid, kThreads, kSmem, st>>>(a);
  LAUNCH_CHECK();
  return CUAPSS_OK;
}

}  // namespace cuapss
