// expand_plan.h -- internal interface of expand_plan.cu.
#pragma once

#include "internal.cuh"

namespace holo {

// SM clocks of the expansion kernels (GB300), per point evaluation of the moments and
// targets kernels and per pair of nodes of the translation.
constexpr double kMomentClocks = 1.6, kTargetClocks = 2.0, kNodePairClocks = 0.3;

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

// The descriptor of a sum (all but its slab) with its buffers taken from `tmp`; share: the
// part of the GPU that it should fill (1 alone, its part of the work in a batch).
ExpandProblem expand_describe(holo_plan_s *p, const ExpandChoice &ch, double sk, double2 *y,
                              double share, ExpandScratch &tmp);
int expand_execute(holo_plan_s *p, const ExpandChoice &ch, double sk, const double *amp,
                   const double *phase, double2 *y, cudaStream_t s);

}  // namespace holo
