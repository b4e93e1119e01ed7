// The host memory, counters and launch of collectives that emulated ranks run over host memory without a ring
// (kernels/sm100/host_exchange.cu).
#pragma once

#include "b200ccl/communicator.h"
#include "core/buffers.h"
#include "kernels/sm100/dev_types.h"

#include <vector>

namespace b200ccl {

class HostExchange {
public:
    // `status`: one record per rank, in mapped host memory.
    HostExchange(int nranks, int device, unsigned long long timeout_ns, std::vector<dev::Status*> status);
    int launch(Collective collective, const CollectiveArgs& args);  // CTAs per rank

private:
    int nranks_, device_;
    unsigned long long timeout_ns_;
    std::vector<dev::Status*> status_;
    MappedBuffer<unsigned char> parts_, results_;
    MappedU64Array given_, done_;
    DeviceBuffer<unsigned long long> tiles_;
    DeviceBuffer<dev::ControlBlock> ctrl_;  // abort word and failure latch of every rank
};

}  // namespace b200ccl
