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

namespace persistent {

template <class TF>
struct PArgs;

// bytes of a launch's work area (D^-1 Av, D^-1 v+, scalars, coefficients)
size_t lockstep_bytes(int n, int num);

// the cooperative launch; a's vectors are zeroed by the caller
template <class TF>
int lockstep_launch(const PArgs<TF>& a, const LockPlan& p, int num, const int* row_off, const int* qb, const int* qe,
                    void* work, double* out, int grid, cudaStream_t s);

template <class TF>
const void* lockstep_kernel();

}  // namespace persistent

}  // namespace culipx
