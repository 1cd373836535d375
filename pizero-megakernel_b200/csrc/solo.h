// Kernels of their own for operators that are launched by themselves.
//
// A program of many stages runs in the persistent kernel (vm_kernel.cuh).  One operator alone pays for what that kernel is built for -
// descriptors fetched from memory, one CTA of 224 KiB per SM, eight warps that change roles, tiles of one SM - and gains nothing from
// it, so the operators that a user launches one at a time have kernels here whose arguments arrive with the launch.  They compute what the
// stage of a program computes; launch_solo decides which operators go this way, and the others run as a program of one stage as before.
#pragma once
#include <cuda_runtime.h>

#include "vm_types.h"

namespace pi0 {

// What every kernel needs beside its operands: where to report a wait that ran out, and how long it may take.
struct SoloGuard {
    VmStatus* status;
    unsigned long long budget_ns;
    unsigned int* counters;      // finished tiles per 128-row band, as the stage of a program leaves them
    int early;                   // let the next launch of the stream prepare while this one runs
};

struct SoloNorm {
    NormParams n;
    SoloGuard guard;
};

cudaError_t launch_solo_norm(const SoloNorm& p, int grid, int groups, cudaStream_t stream);
}  // namespace pi0
