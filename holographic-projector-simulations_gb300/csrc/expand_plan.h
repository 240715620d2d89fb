// expand_plan.h -- internal interface of expand_plan.cu.
#pragma once

#include "internal.cuh"

namespace holo {

// SM clocks of the expansion kernels (GB300): a moments block's 64 sources x 64 target clusters
// alone on an SM (half the rate for each of two), a target item's set-up and its 32 source
// clusters, one pair of nodes of the translation at full load, and per node pair of a thread.
constexpr double kMomentStage = 7000.0, kTargetItem = 5000.0, kTargetGroup = 5000.0,
                 kNodePairClocks = 0.27, kTranslateLatency = 80.0;

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

// Scratch that a sum's target clusters may take per launch, and what it goes down to where the
// device has no room for that.
constexpr size_t kSlabBytes = (size_t)1 << 30, kLeastSlabBytes = (size_t)1 << 24;

// The descriptor of a sum (all but its slab), its sources' amplitudes and phases and its partial
// sums taken from `keep` and the rest, which only its own launches use, from `tmp`; share: the
// part of the GPU that it should fill (1 alone, its part of the work in a batch).
ExpandProblem expand_describe(holo_plan_s *p, const ExpandChoice &ch, double sk, double2 *y,
                              double share, size_t slab_bytes, ExpandScratch &keep,
                              ExpandScratch &tmp);
int expand_execute(holo_plan_s *p, const ExpandChoice &ch, double sk, const double *amp,
                   const double *phase, double2 *y, cudaStream_t s);

}  // namespace holo
