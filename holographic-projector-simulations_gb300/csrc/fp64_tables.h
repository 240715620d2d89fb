// fp64_tables.h -- host-side fill of the fixed-point FP64 kernel's tables.
#pragma once

#include "fp64_fixed.cuh"

namespace holo {
void fill_trig(fixed::TrigEntry *out);    // [fixed::kTrigEntries]
void fill_turns(fixed::TurnWords *out);   // [fixed::kTurnEntries]
void fill_polar(fixed::PolarEntry *out);  // [fixed::kPolarEntries]
}  // namespace holo
