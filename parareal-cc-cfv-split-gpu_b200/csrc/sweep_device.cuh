// sweep_device.cuh -- field lookup and asynchronous-copy helpers shared by the
// sweep kernels (sweep.cu, stream.cu).
#pragma once

#include "ccfv_internal.h"

namespace ccfv {

// Field of tile `tile` (fields sorted by group0): binary search on the
// launch's compact group0 index when it has one (batched launches of
// thousands of fields: a few cache lines instead of one descriptor line per
// probe), else on the descriptors.
__device__ __forceinline__ int find_field(const SweepField *__restrict__ fields,
                                          const int *__restrict__ g0idx, int nfields, int tile) {
  int lo = 0, hi = nfields - 1;
  if (g0idx) {
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(g0idx + mid) <= tile) lo = mid; else hi = mid - 1;
    }
  } else {
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(&fields[mid].group0) <= tile) lo = mid; else hi = mid - 1;
    }
  }
  return lo;
}

// A field's launch time offset (field_active, ccfv_internal.h, says whether
// it takes part in a batched launch).
__device__ __forceinline__ double field_time(const SweepField &f, double toff, int jstep,
                                             int nslice) {
  return toff + jstep * f.t_step + (f.slice < 0 ? nslice * f.t_slice : 0.0);
}

// Input and output of a field in a launch (SweepField::pp): in place, or the
// ping-pong pair of an out-of-place sweep sequence.  Out of place, no CTA
// reads what another CTA of the launch writes.  FieldIo: see launch_sweep.
__device__ __forceinline__ void field_io(const SweepField &f, int jstep, const FieldIo &io,
                                         const void **src, void **dst) {
  void *A = io.data ? io.data : f.data;
  if (!f.pp) {
    *src = A;
    *dst = A;
    return;
  }
  const int s = f.s0 + f.sj * jstep;
  const bool toA = ((s + f.par + (io.mode >> 1)) & 1) != 0;
  const void *in0 = io.in ? io.in : io.data ? io.data : f.in0;
  *src = s == 0 ? in0 : (toA ? f.data2 : A);
  *dst = (io.mode & IO_IN_PLACE) ? const_cast<void *>(*src) : toA ? A : f.data2;
}

__device__ __forceinline__ void cp_async8(void *sdst, const void *gsrc) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async4(void *sdst, const void *gsrc) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all_committed() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async16(void *sdst, const void *gsrc) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}

// x^n (n >= 0) by binary powering, in FP64.
__device__ __forceinline__ double powi(double x, int n) {
  double r = 1.0;
  while (n > 0) {
    if (n & 1) r *= x;
    x *= x;
    n >>= 1;
  }
  return r;
}

}  // namespace ccfv
