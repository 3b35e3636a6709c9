// Chains of short kernels on one stream.  Each lets the next one's blocks
// start while it runs and itself waits, before it touches memory, for the
// kernel before it to be complete; that hides most of a launch's 2 us
// (programmatic dependent launch).  A kernel that is launched plainly, or
// that follows one without chain_begin, behaves as without it.  Measured on
// whole eigensolves: 20^3 15.6 -> 14.8 ms, 46^3 18.1 -> 17.3, 64^3 74.3 ->
// 72.9, largest eigenvalues at 100^3 11.9 -> 11.1.
#pragma once

#include "common.cuh"
#include "launch.h"

namespace spx {

SPX_DEV void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace spx
