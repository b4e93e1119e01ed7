// Collectives whose ranks all live on ONE device: every rank's buffers are this GPU's own memory and one
// stream orders them, so nobody has to wait for anybody inside the kernel.
#pragma once

#include "b200ccl/types.h"

#include <cuda_runtime.h>

#include <cstddef>

namespace b200ccl::kernels {

struct LocalCall {
    Collective collective = Collective::AllReduce;
    DType dtype = DType::Float;
    RedOp redop = RedOp::Sum;  // ignored by all_gather
    int nranks = 1;            // 1: every collective is a copy
    const void* const* in = nullptr;  // nranks pointers each, aligned to the element size at least
    void* const* out = nullptr;
    std::size_t count = 0;     // as in CollectiveArgs::count
    int max_ctas = 0;          // cap on the CTAs of the launch; 0: none
    cudaStream_t stream = nullptr;
};

struct LocalLaunch {  // what a call came to
    int grid = 0;
    int block = 0;
    int pack_bytes = 0;
};

// An input may be the same rank's output (all_reduce); otherwise inputs and outputs do not overlap.
cudaError_t launch_local(const LocalCall& call, LocalLaunch* made);

}  // namespace b200ccl::kernels
