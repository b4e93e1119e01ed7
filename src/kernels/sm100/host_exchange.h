// Collectives through host memory without a ring: two-shot over mapped buffers that every rank can address.
#pragma once

#include "b200ccl/types.h"
#include "kernels/sm100/dev_types.h"

#include <cuda_runtime.h>

namespace b200ccl::dev {

// CTAs per rank, at most. About ten in all keep PCIe busy; more of them disturb one another (4 ranks, 4 MiB: 703 us with two, 725 with
// four, 795 with eight in tiles of 256 rows).
constexpr int host_ctas(int nranks) { return nranks <= 2 ? 4 : (nranks == 3 ? 3 : (nranks < 8 ? 2 : 1)); }
constexpr unsigned kHostChunkRows = 256;  // rows of 512 bytes that a rank's share of a tile has, at most
constexpr unsigned kHostChunkBytes = kHostChunkRows * 512;
constexpr int kHostSlots = 3;

struct HostExchangeArgs {
    const void* in[kMaxRanks];
    void* out[kMaxRanks];
    ControlBlock* ctrl[kMaxRanks];
    Status* status[kMaxRanks];
    unsigned char* parts;        // host: [to][from][cta][slot] chunks, a rank's input for the share of another
    unsigned char* results;      // host: [from][cta][slot] chunks, a rank's share of the result
    unsigned long long* given;   // host: [to][from][cta] tiles whose part has been written
    unsigned long long* done;    // host: [from][cta] tiles whose result has been written
    unsigned long long* tiles;   // device: [rank][cta] tiles of earlier calls
    unsigned long long count;    // the API's count
    unsigned long long timeout_ns;
    float scale;
    int nranks;
    int collective;              // b200ccl::Collective
    unsigned lead;               // 16-byte path: elements by which in[] and out[] are past a 16-byte boundary, all alike
    unsigned long long rows;     // of 512 bytes, of a rank's share (all_reduce) or block
    unsigned first_rows;         // of a CTA's first tile
    int ctas;                    // host_ctas(nranks): what the slots and counters are laid out for
};

}  // namespace b200ccl::dev

namespace b200ccl::kernels {

std::size_t host_parts_bytes(int nranks);
std::size_t host_results_bytes(int nranks);
std::size_t host_given_words(int nranks);
std::size_t host_done_words(int nranks);
std::size_t host_tiles_words(int nranks);

// One cooperative launch that plays every rank (blockIdx.y). Fills in args.rows and what follows. wide as for the ring in clusters.
// `*used`: CTAs per rank.
cudaError_t launch_host_exchange(DType dtype, RedOp op, bool wide, dev::HostExchangeArgs args, cudaStream_t stream, int* used);

}  // namespace b200ccl::kernels
