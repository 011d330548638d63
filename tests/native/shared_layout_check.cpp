// Host check (built by tests/test_shared_layout.py) of what the FP64 kernels' 16-byte asynchronous copies
// rest on: their shared prior table and the ring of the row above behind it start on 16-byte boundaries,
// whatever else the kernel keeps in shared memory, and so does every warp's scratch row.
#include "warp_emu_shim.h"

#include <cstddef>

#include "../../rovaca_b200/csrc/phmm_device64.cuh"
#include "../../rovaca_b200/csrc/phmm_plan.h"

using namespace phmm;

struct Neighbour {
    double before;
    PriorTable64<kMaxK> tab;
};
static_assert(alignof(PriorTable64<kMaxK>) == 16 && alignof(PriorTable64<1>) == 16, "table");
static_assert(offsetof(Neighbour, tab) % 16 == 0, "table next to another variable");
static_assert(sizeof(PriorTable64<kMaxK>) == prior_table_size<kMaxK>() * sizeof(double), "no padding");
static_assert(kTabClasses * kMaxK * kWarp * sizeof(double) % 16 == 0, "ring");
static_assert((uint64_t)PlanLimits().max_stream_multi * 24 % 16 == 0, "scratch row");

int main() { return 0; }
