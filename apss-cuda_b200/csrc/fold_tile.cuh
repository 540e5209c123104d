// Device helpers shared by the folded tile kernels.
#pragma once

#include "fold.cuh"
#include "ptx.cuh"

namespace cuapss {

// Bounded wait (kWaitLimitNs of device time) that also gives up when another
// role raised the abort flag.
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

// Raises the abort flag and reports the timeout.
__device__ __forceinline__ void give_up(int* err, volatile int* abort) {
  if (!*abort) {
    *abort = 1;
    atomicOr(err, kErrTimeout);
  }
}

// wait_abort for a whole warp: every lane waits and the warp takes one answer.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort,
                                          int* err, bool live) {
  bool got = live ? wait_abort(bar, parity, abort) : true;
  got = __all_sync(0xffffffffu, got);
  if (live && !got && (threadIdx.x & 31) == 0) give_up(err, abort);
  return live && got;
}

// The next unit of a CTA's producer (the two round trips to L2 overlap: one
// after the other they took 9 of the 213 us of a one-row index query).
__device__ __forceinline__ int next_unit(const FoldTileArgs& A) {
  const int u = atomicAdd(A.unit_counter, 1);
  if (A.give_up_at <= 0) return u;
  const unsigned long long found = *const_cast<const volatile unsigned long long*>(A.cand_count);
  return found > (unsigned long long)A.give_up_at ? A.nunits : u;
}

// Appends a warp's held candidates to the list: one reservation for up to
// kHits of them. True: the join is given up.
__device__ __forceinline__ bool flush_hits(const FoldTileArgs& A, const uint64_t* hits, int n,
                                           int lane) {
  __syncwarp();
  unsigned long long w = 0;
  if (lane == 0) w = atomicAdd(A.cand_count, (unsigned long long)n);
  w = __shfl_sync(0xffffffffu, w, 0);
  for (int k = lane; k < n; k += 32)
    if ((int64_t)w + k < A.cand_cap) A.cand[w + k] = hits[k];
  __syncwarp();
  return A.give_up_at > 0 && (int64_t)w + n > A.give_up_at;
}

}  // namespace cuapss
