// expand_plan.h -- internal interface of expand_plan.cu.
#pragma once

#include "internal.cuh"

namespace holo {

// SM clocks of the expansion kernels (GB300), per point evaluation of the moments and
// targets kernels and per pair of nodes of the translation; seconds of their launches.
constexpr double kMomentClocks = 1.6, kTargetClocks = 2.0, kNodePairClocks = 0.3;
constexpr double kExpandOverhead = 30e-6, kPairOverhead = 10e-6;

// One device buffer for all of a sum's scratch: a first pass over the takes adds up the size,
// a second one hands out the addresses.
struct ExpandScratch {
  unsigned char *base = nullptr;
  size_t bytes = 0;
  template <typename T>
  T *take(size_t count) {
    T *p = reinterpret_cast<T *>(base + bytes);
    bytes += (count * sizeof(T) + 255) / 256 * 256;
    return base ? p : nullptr;
  }
};

// The descriptor of a sum (all but its slab) with its buffers taken from `tmp`.
ExpandProblem expand_describe(holo_plan_s *p, const ExpandChoice &ch, double sk, double2 *y,
                              ExpandScratch &tmp);
int expand_execute(holo_plan_s *p, const ExpandChoice &ch, double sk, const double *amp,
                   const double *phase, double2 *y, cudaStream_t s);

}  // namespace holo
