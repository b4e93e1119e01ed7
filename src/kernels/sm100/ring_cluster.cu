// Ring collectives of ranks that share a GPU, through distributed shared memory.
//
// The schedule is that of ring_simple.cu: slices go round the ring through a FIFO in the receiver's memory, a rank waits for a
// slice, combines it with its own input, passes it on and returns the slot. Between GPUs that memory is global and the
// hand-over is a release and an acquire of step counters, which takes 3.4 us per hop on one B200 (1.2 to release, 1 to see
// the counter, 1.2 to load the slice). Here the CTAs of a channel, one per rank, are a thread block cluster: the receiver's
// memory is its shared memory, a slice goes there with st.async, whose bytes an mbarrier of the receiver counts, and a slot is
// returned by an arrival on an mbarrier of the sender, behind a fence for shared memory only. No counter is polled in global memory.
//
// Every warp is a ring of its own (a unit): it talks to the warps of the same index in the neighbours' CTAs only, so that
// there is no barrier in the loop, and an SM's sixteen warps hide one another's hops (0.35 us for a slice of 512 bytes). They
// come as four CTAs of four warps: a cluster lies within one GPC, and of small CTAs more clusters fit (8 ranks, one CTA of 16 warps
// per SM 15 clusters on 120 SMs, now 71 that fill 142: 64 MiB 301 -> 259 us; 7 ranks 292 -> 230; two CTAs of 8 warps 275 and 240). The local
// input of the next step is loaded before the wait for the neighbour. A slice is 1, 2, 4 or 8 rows of 32 vectors; the message is
// cut so that all slices but its last ones are full and move without a condition per vector.
//
// Bound by the hops up to about 1 MiB, then by distributed shared memory (4.0-4.4 TB/s into neighbours, 5.3 in pairs; st.async,
// plain remote stores and bulk copies alike). float sum, us with FIFOs in global memory and two groups of eight warps -> here: 4
// ranks, 4 KiB 22.4 -> 8.2, 1 MiB 28.9 -> 10.2, 16 MiB 58.6 -> 35.8, 64 MiB 199 -> 124; 2 ranks, 64 MiB 133 -> 51; 8 ranks, 4 KiB 36.9 ->
// 12.3, 64 MiB 407 -> 261; bf16, 4 ranks, 16 MiB of views that start off a vector 219 -> 39, reduce_scatter in ragged blocks of 4 MiB
// 128 -> 31. Slots of 3 slices instead of 2, or slices of 4 rows for all sizes, are slower.
//
// Every wait is bounded. The launch is cooperative, as all launches whose CTAs wait for one another.
#include "kernels/sm100/ring_cluster.h"

#include "kernels/sm100/sync.cuh"
#include "kernels/sm100/tma.cuh"
#include "kernels/sm100/vec.cuh"
#include "sched/ring_geometry.h"

#include <algorithm>
#include <type_traits>

namespace b200ccl::kernels {

using namespace b200ccl::dev;

namespace {

using u64 = unsigned long long;

constexpr int kWarps = 4, kThreads = kWarps * 32, kCtasPerSm = 4;
constexpr int kSlots = 2;                 // slices that a unit's FIFO holds
constexpr unsigned kRowBytes = 32 * 16;   // what a warp moves at a time
// Rows of a slice (kRows below): 8 move most, fewer keep more warps busy in small messages.
constexpr int kMostRows = 8;
constexpr unsigned kFifoBytes = kWarps * kSlots * kMostRows * kRowBytes;

enum StepFlags : unsigned { kRecv = 1u, kLocal = 2u, kSend = 4u, kCopyOut = 8u, kScale = 16u };

struct Step {
    unsigned flags;
    unsigned n;         // elements of the slice
    u64 in_at, out_at;  // where it lies in the local input and output
};

__device__ __forceinline__ unsigned of_rank(unsigned smem, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem), "r"(rank));
    return a;
}
__device__ __forceinline__ uint4 ld_slot16(unsigned smem) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(smem) : "memory");
    return v;
}
// 16 bytes into the next rank's FIFO; its mbarrier counts them.
__device__ __forceinline__ void st_slot16(unsigned remote, const uint4& v, unsigned remote_bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1,%2,%3,%4}, [%5];" ::"r"(remote), "r"(v.x),
                 "r"(v.y), "r"(v.z), "r"(v.w), "r"(remote_bar)
                 : "memory");
}
// The one arrival that a slice's phase needs, with the bytes that make it complete; in any order with the stores.
__device__ __forceinline__ void announce(unsigned remote_bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cluster.b64 _, [%0], %1;" ::"r"(remote_bar), "r"(bytes) : "memory");
}
// Hands a slot of this CTA back to the rank that fills it, whose wait acquires at cluster scope. What the warp has read from the slot
// before is ordered before everything that rank does after its wait: __syncwarp() orders the lanes' reads before the fence, and the
// fence releases at cluster scope what was done to this CTA's shared memory. It does not wait for the stores to the output, as an arrival
// that releases everything does (float sum, us, here / so: 4 ranks, 4 KiB 8.2 / 10.3, 16 MiB 35.8 / 43.0; 8 ranks, 64 MiB 261 / 319).
__device__ __forceinline__ void return_slot(unsigned remote_bar, unsigned lane) {
    __syncwarp();
    if (lane == 0) {
        asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory");
        asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote_bar) : "memory");
    }
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

template <typename T, typename Op, bool kWide, int kRows>
__global__ void __launch_bounds__(kThreads, kCtasPerSm) ring_cluster_kernel(const __grid_constant__ RingClusterArgs a) {
    constexpr int kElems = 16 / sizeof(T);
    constexpr unsigned kRow = 32u * kElems, kSlice = kRows * kRow, kSliceBytes = kRows * kRowBytes;  // elements, elements, bytes
    extern __shared__ __align__(128) unsigned char fifo[];
    __shared__ u64 full[kWarps][kSlots], empty[kWarps][kSlots];
    __shared__ unsigned failed;
    const int n = a.nranks, r = (int)blockIdx.y;  // the cluster is 1 x nranks: the rank is the CTA's rank in it
    const unsigned warp = threadIdx.x / 32u, lane = threadIdx.x & 31u;
    const unsigned next = (unsigned)(r + 1 == n ? 0 : r + 1), prev = (unsigned)(r == 0 ? n - 1 : r - 1);
    if (threadIdx.x < kWarps * kSlots) {
        mbar_init(&full[0][0] + threadIdx.x, 1u);
        mbar_init(&empty[0][0] + threadIdx.x, 1u);
    }
    if (threadIdx.x == 0) failed = 0u;
    mbar_fence_init();
    cluster_sync();

    const unsigned unit = warp * gridDim.x + blockIdx.x;  // few units: one per cluster
    const unsigned slots = smem_addr(fifo) + warp * (kSlots * kSliceBytes) + lane * 16u, next_slots = of_rank(slots, next);
    const unsigned full_bar = smem_addr(&full[warp][0]), next_full = of_rank(full_bar, next);
    const unsigned empty_bar = smem_addr(&empty[warp][0]), prev_empty = of_rank(empty_bar, prev);
    unsigned sent = 0, received = 0;  // slices

    const T* in = static_cast<const T*>(a.in[r]);
    T* out = static_cast<T*>(a.out[r]);
    const unsigned lead = kWide ? a.lead : 0u;
    in -= lead;  // aligned; the `lead` elements before the buffer are never accessed
    out -= lead;

    const u64 total = a.count + lead;  // elements from the boundary on
    const bool reduces = a.collective != (int)Collective::AllGather, scatters = a.collective == (int)Collective::ReduceScatter;
    const bool both = reduces && !scatters;
    // A unit takes the windows unit, unit + units, ...: n slices of the message (all_reduce), or one slice of every block. All
    // slices but the last ones of a message are full.
    const u64 window = both ? (u64)n * kSlice : kSlice;
    const int steps = both ? 2 * n - 1 : n;

    auto step_at = [&](u64 w0, int j) {
        Step s;
        if (reduces) {
            if (j == 1) s.flags = kLocal | kSend;
            else if (j < n) s.flags = kRecv | kLocal | kSend;
            else if (scatters) s.flags = kRecv | kLocal | kCopyOut | kScale;  // own block
            else if (j == n) s.flags = kRecv | kLocal | kSend | kCopyOut | kScale;  // pivot: final value → output and onwards
            else s.flags = j < steps ? kRecv | kSend | kCopyOut : kRecv | kCopyOut;
        } else {
            s.flags = j == 1 ? kLocal | kSend | kCopyOut : (j < n ? kRecv | kSend | kCopyOut : kRecv | kCopyOut);
        }
        int k = reduces ? r - j : r + 1 - j;  // chunk (all_reduce) or block
        if (k < 0) k += n;
        if (k < 0) k += n;
        u64 at = w0;
        if (both) {
            at += (u64)k * kSlice;
            s.in_at = s.out_at = at;
        } else {
            const u64 block = (u64)k * a.count + w0;
            s.in_at = scatters ? block : w0;
            s.out_at = scatters ? w0 : block;
        }
        s.n = (unsigned)ring::clamp_elems(kSlice, total, at);
        return s;
    };

    // Vector u of a lane: kElems elements behind one another (16-byte path), or 32 apart, so that a warp's accesses are
    // contiguous; which of them exist.
    auto first_of = [&](int u) { return kWide ? (unsigned)(u * 32 + lane) * kElems : (unsigned)(u * 32 * kElems) + lane; };
    constexpr unsigned kStride = kWide ? 1u : 32u;
    auto load_some = [&](const T* base, u64 at, unsigned i0, unsigned n_, uint4& v) {
        T t[kElems];
#pragma unroll
        for (int e = 0; e < kElems; ++e) {
            const unsigned i = i0 + e * kStride;
            t[e] = Elem<T>::from_f(0.0f);
            if (i < n_ && (!kWide || at + i >= lead)) t[e] = Narrow<T>::load(base, at + i);
        }
        v = *reinterpret_cast<const uint4*>(t);
    };
    auto store_some = [&](T* base, u64 at, unsigned i0, unsigned n_, const uint4& v) {
        T t[kElems];
        *reinterpret_cast<uint4*>(t) = v;
#pragma unroll
        for (int e = 0; e < kElems; ++e) {
            const unsigned i = i0 + e * kStride;
            if (i < n_ && (!kWide || at + i >= lead)) base[at + i] = t[e];
        }
    };
    auto whole = [&](u64 at, unsigned i0, unsigned n_) { return kWide && i0 + kElems <= n_ && at + i0 >= lead; };

    uint4 mine[kRows], got[kRows];
    // A slice is up to kRows rows of a warp. Of a full slice every row is moved without a condition.
    auto is_full = [&](const Step& s, u64 at) { return s.n == kSlice && (!kWide || at >= lead); };
    auto load_local = [&](const Step& s) {
        const T* p = in + s.in_at;
        if (is_full(s, s.in_at)) {
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                if constexpr (kWide) {
                    mine[u] = ld16_stream(reinterpret_cast<const uint4*>(p) + u * 32 + lane);
                } else {
                    T t[kElems];
#pragma unroll
                    for (int e = 0; e < kElems; ++e) t[e] = Narrow<T>::load(p, first_of(u) + e * kStride);
                    mine[u] = *reinterpret_cast<const uint4*>(t);
                }
            }
            return;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            if (u * kRow >= s.n) break;
            const unsigned i0 = first_of(u);
            if (i0 >= s.n) continue;
            if (whole(s.in_at, i0, s.n)) mine[u] = ld16_stream(reinterpret_cast<const uint4*>(p + i0));
            else load_some(in, s.in_at, i0, s.n, mine[u]);
        }
    };
    // One slice, up to the slot of the next rank; false when a wait gave up.
    auto exchange = [&](const Step& s, auto is_full_slice) {
        constexpr bool kFull = decltype(is_full_slice)::value;
        auto over = [&](int u) { return !kFull && u * kRow >= s.n; };
        auto has = [&](int u) { return kFull || first_of(u) < s.n; };
        if (s.flags & kRecv) {
            const unsigned slot = received % kSlots;
            if (!wait_cluster_phase(full_bar + slot * 8u, (received / kSlots) & 1u, &failed, a.ctrl[r], a.timeout_ns, a.status[r], prev, 10u, received)) return false;
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                if (over(u)) break;
                if (has(u)) got[u] = ld_slot16(slots + slot * kSliceBytes + u * 512u);
            }
            const bool scaled = (s.flags & kScale) && a.scale != 1.0f, local = s.flags & kLocal;
            if (local || scaled) {
#pragma unroll
                for (int u = 0; u < kRows; ++u) {
                    if (over(u)) break;
                    if (!has(u)) continue;
                    float acc[kElems], f[kElems];
                    Wide<T>::unpack(got[u], acc);
                    if (local) {
                        Wide<T>::unpack(mine[u], f);
#pragma unroll
                        for (int e = 0; e < kElems; ++e) acc[e] = Op::apply(f[e], acc[e]);
                    }
                    if (scaled) {
#pragma unroll
                        for (int e = 0; e < kElems; ++e) acc[e] *= a.scale;
                    }
                    got[u] = Wide<T>::pack(acc);
                }
            }
            return_slot(prev_empty + slot * 8u, lane);
            ++received;
        } else {
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                if (over(u)) break;
                got[u] = mine[u];
            }
        }
        if (s.flags & kSend) {
            const unsigned slot = sent % kSlots;
            if (sent >= kSlots &&
                !wait_cluster_phase(empty_bar + slot * 8u, (sent / kSlots - 1u) & 1u, &failed, a.ctrl[r], a.timeout_ns, a.status[r], next, 11u, sent))
                return false;
            unsigned lanes = kRows * 32u;  // 16-byte vectors of the slice, all lanes' together
            if (!kFull) lanes = kWide ? (s.n + kElems - 1u) / kElems : s.n / (32u * kElems) * 32u + min(s.n % (32u * kElems), 32u);
            if (lane == 0) announce(next_full + slot * 8u, lanes * 16u);
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                if (over(u)) break;
                if (has(u)) st_slot16(next_slots + slot * kSliceBytes + u * 512u, got[u], next_full + slot * 8u);
            }
            ++sent;
        }
        return true;
    };
    auto store_out = [&](const Step& s) {
        T* p = out + s.out_at;
        if (is_full(s, s.out_at)) {
#pragma unroll
            for (int u = 0; u < kRows; ++u) {
                if constexpr (kWide) {
                    st16(reinterpret_cast<uint4*>(p) + u * 32 + lane, got[u]);
                } else {
                    T t[kElems];
                    *reinterpret_cast<uint4*>(t) = got[u];
#pragma unroll
                    for (int e = 0; e < kElems; ++e) p[first_of(u) + e * kStride] = t[e];
                }
            }
            return;
        }
#pragma unroll
        for (int u = 0; u < kRows; ++u) {
            if (u * kRow >= s.n) break;
            const unsigned i0 = first_of(u);
            if (i0 >= s.n) continue;
            if (whole(s.out_at, i0, s.n)) st16(reinterpret_cast<uint4*>(p + i0), got[u]);
            else store_some(out, s.out_at, i0, s.n, got[u]);
        }
    };

    const u64 stride = window * (unsigned)a.units;
    u64 w0 = unit < (unsigned)a.units ? window * unit : total;
    int j = 1;
    bool more = w0 < total, ok = true;
    Step s{};
    if (more) {
        s = step_at(w0, j);
        if (s.flags & kLocal) load_local(s);
    }
    while (more) {
        if (s.n != 0) {  // an empty slice: neither side waits or sends
            if (!(s.n == kSlice ? exchange(s, std::true_type{}) : exchange(s, std::false_type{}))) {
                ok = false;
                break;
            }
        }
        const Step done = s;
        if (++j > steps) {
            j = 1;
            w0 += stride;
        }
        more = w0 < total;
        if (more) {
            s = step_at(w0, j);
            if (s.flags & kLocal) load_local(s);
        }
        if (done.flags & kCopyOut) store_out(done);
    }
    // No CTA leaves while a neighbour may still store into its shared memory: every slice that was sent has been waited for,
    // unless a wait gave up somewhere in the cluster. Every CTA learns of that and waits for what is under way.
    if (!ok && lane < (unsigned)n) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(of_rank(smem_addr(&failed), lane)), "r"(1u) : "memory");
    __syncwarp();
    cluster_sync();
    if (*static_cast<volatile unsigned*>(&failed) != 0u) {
        for (unsigned k = received; k < received + kSlots; ++k) drain_cluster_phase(full_bar + (k % kSlots) * 8u, (k / kSlots) & 1u);
        __syncwarp();
        cluster_sync();
    }
}

using Kernel = void (*)(RingClusterArgs);

cudaLaunchConfig_t configure(int nranks, int clusters, cudaStream_t stream, cudaLaunchAttribute (&attrs)[2]) {
    attrs[0].id = cudaLaunchAttributeClusterDimension;
    attrs[0].val.clusterDim.x = attrs[0].val.clusterDim.z = 1;
    attrs[0].val.clusterDim.y = static_cast<unsigned>(nranks);
    attrs[1].id = cudaLaunchAttributeCooperative;
    attrs[1].val.cooperative = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(static_cast<unsigned>(clusters), static_cast<unsigned>(nranks), 1);
    config.blockDim = dim3(kThreads, 1, 1);
    config.dynamicSmemBytes = kFifoBytes;
    config.stream = stream;
    config.attrs = attrs;
    config.numAttrs = 2;
    return config;
}

template <typename T, typename Op>
Kernel pick(bool wide, int rows) {
    switch (rows) {
        case 1: return wide ? ring_cluster_kernel<T, Op, true, 1> : ring_cluster_kernel<T, Op, false, 1>;
        case 2: return wide ? ring_cluster_kernel<T, Op, true, 2> : ring_cluster_kernel<T, Op, false, 2>;
        case 4: return wide ? ring_cluster_kernel<T, Op, true, 4> : ring_cluster_kernel<T, Op, false, 4>;
        default: return wide ? ring_cluster_kernel<T, Op, true, 8> : ring_cluster_kernel<T, Op, false, 8>;
    }
}

template <typename T>
Kernel pick_op(RedOp op, bool wide, int rows) {
    switch (op) {
        case RedOp::Sum:
        case RedOp::Avg: return pick<T, OpAdd>(wide, rows);
        case RedOp::Max: return pick<T, OpMax>(wide, rows);
        case RedOp::Min: return pick<T, OpMin>(wide, rows);
    }
    return nullptr;
}

}  // namespace

int ring_cluster_threads() { return kThreads; }
int ring_clusters_per_channel() { return kCtasPerSm; }

int ring_cluster_capacity(int nranks) {
    const Kernel kernel = pick<float, OpAdd>(true, kMostRows);  // every instance runs kCtasPerSm: its FIFOs and registers see to that
    int clusters = 0;
    cudaLaunchAttribute attrs[2];
    const cudaLaunchConfig_t config = configure(nranks, 1, nullptr, attrs);
    if (cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, kFifoBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return clusters;
}

cudaError_t launch_ring_cluster(DType dtype, RedOp op, bool wide, RingClusterArgs args, int clusters, cudaStream_t stream, int* used) {
    if (args.nranks < 2 || args.nranks > kMaxRanks || clusters < 1) return cudaErrorInvalidValue;
    // Rows per slice: all warps together move the same bytes whatever it is, but a unit takes its windows one after the other,
    // and every further one adds a round of hops, each as long as about kHopRows rows of every warp. The fewest rounds, then
    // the shortest slices.
    constexpr u64 kHopRows = 3;
    const u64 bytes = (args.count + args.lead) * dtype_size(dtype), most_units = static_cast<u64>(clusters) * kWarps;
    const u64 row = kRowBytes * (args.collective == static_cast<int>(Collective::AllReduce) ? static_cast<u64>(args.nranks) : 1);
    int rows = 0;
    u64 best = 0, windows = 0;
    for (int v = 1; v <= kMostRows; v *= 2) {
        const u64 w = ring::div_up(bytes, row * v), cost = w * v + ring::div_up(w, most_units) * kHopRows * most_units;
        if (rows == 0 || cost < best) {
            rows = v;
            best = cost;
            windows = w;
        }
    }
    args.units = static_cast<int>(std::min(std::max<u64>(windows, 1), most_units));
    clusters = std::min(clusters, args.units);
    Kernel kernel = nullptr;
    switch (dtype) {
        case DType::Float: kernel = pick_op<float>(op, wide, rows); break;
        case DType::Float16: kernel = pick_op<__half>(op, wide, rows); break;
        case DType::BFloat16: kernel = pick_op<__nv_bfloat16>(op, wide, rows); break;
    }
    if (kernel == nullptr) return cudaErrorInvalidValue;
    cudaError_t st = cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, kFifoBytes);
    if (st != cudaSuccess) return st;
    cudaLaunchAttribute attrs[2];
    const cudaLaunchConfig_t config = configure(args.nranks, clusters, stream, attrs);
    *used = clusters;
    return cudaLaunchKernelEx(&config, kernel, args);
}

}  // namespace b200ccl::kernels
