// Ring collectives of emulated ranks: the ranks of a channel are one thread block cluster, and its FIFOs lie in distributed
// shared memory.
#pragma once

#include "b200ccl/types.h"
#include "kernels/sm100/dev_types.h"

#include <cuda_runtime.h>

namespace b200ccl::dev {

struct RingClusterArgs {
    const void* in[kMaxRanks];
    void* out[kMaxRanks];
    ControlBlock* ctrl[kMaxRanks];
    Status* status[kMaxRanks];
    unsigned long long count;       // the API's count
    unsigned long long timeout_ns;
    float scale;
    int nranks;
    int collective;  // b200ccl::Collective
    int units;       // warps per rank that have a part of the message
    unsigned lead;   // 16-byte path: elements by which in[] and out[] are past a 16-byte boundary, all alike
};

}  // namespace b200ccl::dev

namespace b200ccl::kernels {

// Clusters of `nranks` CTAs that are resident at once on the current device; 0 when it cannot be told.
int ring_cluster_capacity(int nranks);
int ring_cluster_threads();  // of a CTA
// Clusters that make a channel: as many warps of every rank as a channel of ring_simple.cu has, on as many SMs.
int ring_clusters_per_channel();

// One cooperative launch of at most `clusters` clusters. wide: 16-byte accesses (all_reduce: buffers aligned alike modulo 16, args.lead
// elements past it; reduce_scatter and all_gather: buffers and every block 16-byte aligned), else element by element.
// `*used`: the clusters that were launched.
cudaError_t launch_ring_cluster(DType dtype, RedOp op, bool wide, dev::RingClusterArgs args, int clusters, cudaStream_t stream, int* used);

}  // namespace b200ccl::kernels
