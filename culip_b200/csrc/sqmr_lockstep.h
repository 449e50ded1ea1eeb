// The batched solve on the whole grid (sqmr_lockstep.cu).
#pragma once

#include "device.h"

namespace culipx {

// Work units of a batch over a two-level pattern: level-0 rows in chunks of
// one system (first position in the level list, rows, system) and level-1
// block rows (block row, first row, rows, system).
struct LockPlan {
    int chunks = 0, tiles = 0;  // both 0: the batch has no such plan
    DeviceBuffer units;         // int4: chunks, tiles
    bool use = false;           // the batch's shape is one that gains by it
};

// A batch leaves the whole grid once none of its unfinished systems has more
// rows.  A CTA of its own takes a system of 450 rows 17 us an iteration, one of
// 3000 rows 43; the whole grid took 31 to 53 for 20 to 100 such systems.
constexpr int kLockRows = 3000;

namespace persistent {

template <class TF>
struct PArgs;
struct BatchArgs;

// bytes of a launch's work area (D^-1 Av, D^-1 v+, scalars, coefficients)
size_t lockstep_bytes(int n, int num);

// the cooperative launch and the launch that finishes what it leaves; a's
// vectors are zeroed by the caller, bt's counter here
template <class TF>
int lockstep_launch(const PArgs<TF>& a, const LockPlan& p, const BatchArgs& bt, void* work, int grid, int rest_grid,
                    cudaStream_t s);

template <class TF>
const void* lockstep_kernel();

}  // namespace persistent

}  // namespace culipx
