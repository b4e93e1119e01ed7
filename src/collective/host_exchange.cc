#include "collective/host_exchange.h"

#include "core/check.h"
#include "core/numa.h"
#include "kernels/sm100/host_exchange.h"

#include <cstdint>
#include <cstring>
#include <utility>

namespace b200ccl {

HostExchange::HostExchange(int nranks, int device, unsigned long long timeout_ns, std::vector<dev::Status*> status)
    : nranks_(nranks), device_(device), timeout_ns_(timeout_ns), status_(std::move(status)) {
    const int node = numa::gpu_node(device);
    parts_.reset(kernels::host_parts_bytes(nranks), node);
    results_.reset(kernels::host_results_bytes(nranks), node);
    given_.reset(kernels::host_given_words(nranks), node);
    done_.reset(kernels::host_done_words(nranks), node);
    tiles_.reset(device, kernels::host_tiles_words(nranks));
    tiles_.zero();
    ctrl_.reset(device, static_cast<std::size_t>(nranks));
    ctrl_.zero();
    log_info("host exchange: %zu bytes of parts, %zu of results", kernels::host_parts_bytes(nranks), kernels::host_results_bytes(nranks));
}

int HostExchange::launch(Collective collective, const CollectiveArgs& args) {
    const std::size_t esz = dtype_size(args.dtype);
    dev::HostExchangeArgs a;
    std::memset(&a, 0, sizeof(a));
    std::uintptr_t differ = 0;
    const auto first = reinterpret_cast<std::uintptr_t>(args.send_buffers[0]);
    for (int r = 0; r < nranks_; ++r) {
        a.in[r] = args.send_buffers[r];
        a.out[r] = args.recv_buffers[r];
        a.ctrl[r] = ctrl_.get() + r;
        a.status[r] = status_[r];
        differ |= (reinterpret_cast<std::uintptr_t>(a.in[r]) ^ first) | (reinterpret_cast<std::uintptr_t>(a.out[r]) ^ first);
    }
    a.parts = parts_.get();
    a.results = results_.get();
    a.given = given_.get();
    a.done = done_.get();
    a.tiles = tiles_.get();
    a.count = args.count;
    a.timeout_ns = timeout_ns_;
    a.scale = args.redop == RedOp::Avg ? 1.0f / static_cast<float>(nranks_) : 1.0f;
    a.nranks = nranks_;
    a.collective = static_cast<int>(collective);
    // 16-byte accesses: an all_reduce of buffers that are aligned alike; the blocks of the others must all be aligned.
    const bool alike = (differ & 15u) == 0;
    const bool wide = alike && (collective == Collective::AllReduce || ((first & 15u) == 0 && (args.count * esz) % 16 == 0));
    if (wide) a.lead = static_cast<unsigned>((first & 15u) / esz);
    int used = 0;
    DeviceGuard guard(device_);
    B2_CUDA(kernels::launch_host_exchange(args.dtype, args.redop, wide, a, args.streams[0], &used));
    return used;
}

}  // namespace b200ccl
