// Direct collectives for sm_100a: AllReduce (one-shot, two-shot, NVLS), ReduceScatter and
// AllGather as single kernels that load and store peer GPUs' memory over NVLink / NVSwitch.
//
// What is fused into the one launch per rank: the cross-GPU barriers, the peer loads, the fp32
// widening and accumulation, the avg 1/N scale, the rounding, the stores to peers (or the
// multimem broadcast), and, for buffers that peers cannot address, the copy into and out of the
// staging arena. No separate elementwise kernel runs.
//
// Parity: replaces nano-nccl's only kernel, ring_simple_kernel (src/kernels/
// ring_simple_kernel.cuh:1118-1237), whose 2(N-1) neighbour hops become two hops (pull the own
// shard from every peer, push the result to every peer) or one (every rank pulls everything).
// The reference's pivot step "reduce + scale + write output + forward" (kernel:433-481) is the
// store_all branch below. Its 4-CTA launch (communicator.cu:1094-1095) becomes a grid sized by
// the tuner.
#include "kernels/sm100/direct_collectives.h"

#include "kernels/sm100/sync.cuh"
#include "kernels/sm100/vec.cuh"

#include <type_traits>

namespace b200ccl::kernels {

using namespace b200ccl::dev;

namespace {

using u64 = unsigned long long;

// A kernel parameter is one rank's arguments, or what all emulated ranks share (OneGpu), or, in the checking build, the
// arguments of every emulated rank (LoopPack), of which the CTA picks the one of rank blockIdx.y.
template <typename A>
__device__ __forceinline__ const A& select_args(const A& one) { return one; }
template <typename A>
__device__ __forceinline__ const A& select_args(const LoopPack<A>& all) { return all.r[blockIdx.y]; }
template <typename A>
__device__ __forceinline__ const A& select_args(const OneGpu<A>& all) { return all.a; }
template <typename A>
constexpr bool kAllRanksHere = false;
template <typename A>
constexpr bool kAllRanksHere<OneGpu<A>> = true;

// Emulated ranks are part of one launch: what it finds in memory is every rank's input and its end is every rank's, and no
// rank reads what another one writes (rank r alone reads and writes shard r). So they have nothing to meet for; the launch
// need not be cooperative nor resident all at once, a rank has one CTA for every 8 KiB that it stores to each output, and the launch is a programmatic
// dependent of the one before. As one cooperative launch of CTAs that stayed and met over flags, kernels also followed one
// another only every 2.05 us. Meeting in thread block clusters (1 x ranks) costs little in small calls, but leaves too few
// loads in flight in large ones. bf16 two-shot, us before / in clusters of 512 threads / now: 4 ranks, 4 KiB 6.1 / 3.1 / 3.1,
// 2 MiB 8.2 / 5.7 / 3.7, 8 MiB 16.4 / 14.4 / 11.7 (5.7 TB/s), 256 MiB 346 / 337 / 311 (6.9 TB/s); 8 ranks, 8 MiB 28.5 / 32.5 / 22.5, 256 MiB
// 649 / 870 / 625; one-shot, which is bound by reading every input once per rank through L2: 8 ranks, 4 MiB 36.6 / 71.2 / 23.0.

// Starts a call, behind the launch before it, on `bytes` of the rank's share. The next launch may come at once; where a rank has fewer
// CTAs than take 32 bytes per thread (the caller caps them), only when this one runs: else several launches wait on the SMs, and
// those of one come to lie two on an SM with others idle (two-shot, 4 ranks, 8 MiB, 16 CTAs each: 15.5 us, 23.4 us when the next comes at
// once).
template <typename ParamT>
__device__ __forceinline__ void begin_call(u64 bytes) {
    if constexpr (kAllRanksHere<ParamT>) {
        const bool loops = (u64)gridDim.x * blockDim.x * 32 < bytes;
        if (!loops) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (loops) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
}

// Where ranks on GPUs of their own meet over flags; `epoch` counts the meetings. False when a wait gave up.
template <typename ParamT, typename A>
__device__ __forceinline__ bool meet(const A& a, int rank, int n, u64& epoch, unsigned where, u64 plan_hash) {
    if constexpr (kAllRanksHere<ParamT>) {
        return true;
    } else {
        ++epoch;
        return cta_barrier_all_ranks(a.ctrl, rank, n, epoch, a.timeout_ns, a.status, where, plan_hash);
    }
}

// How many meetings this CTA has been through.
template <typename ParamT>
__device__ __forceinline__ u64 read_epoch(const ControlBlock* own) {
    if constexpr (kAllRanksHere<ParamT>) {
        return 0;
    } else {
        __shared__ u64 s_epoch;
        if (threadIdx.x == 0) s_epoch = own->epoch[blockIdx.x];
        __syncthreads();
        return s_epoch;
    }
}

// Copies the packs first, first+stripe, ... below len, four loads in flight per thread. One side is
// the caller's own buffer (16-byte aligned at most), the other the staging arena.
template <typename P, bool kFromUser>
__device__ __forceinline__ void copy_stripes(void* dst, u64 dst0, const void* src, u64 src0, u64 first, u64 len, u64 stripe) {
    for (u64 j = first; j < len; j += stripe * 4) {
        typename P::Raw v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (j + (u64)u * stripe < len) {
                if constexpr (kFromUser) v[u] = P::load_user(src, src0 + j + (u64)u * stripe);
                else v[u] = P::load(src, src0 + j + (u64)u * stripe);
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (j + (u64)u * stripe < len) {
                if constexpr (kFromUser) P::store(dst, dst0 + j + (u64)u * stripe, v[u]);
                else P::store_user(dst, dst0 + j + (u64)u * stripe, v[u]);
            }
        }
    }
}

// Packs in flight per thread and peer: fewer ranks, or narrower packs, leave room for more.
template <int N, int kPackBytes>
struct UnrollFor {
    static constexpr int k16 = N == 0 ? 1 : (N >= 8 ? 1 : (N >= 4 ? 2 : 4));
    static constexpr int value = kPackBytes == 32 ? (k16 > 1 ? k16 / 2 : 1) : k16;
};

#if defined(B200CCL_DEBUG_BOUNDS)
// Checking builds: an index beyond the extent that the host passed is recorded (first one wins) and
// the access is skipped; the kernel still runs to its end, so no wait is left hanging.
#define B2_IN_BOUNDS(index, extent, where_)                                                                    \
    ((extent) == 0ull || (index) < (extent) ||                                                                \
     (report_failure(a.status, own, nullptr, 0, kStatusBadArgs, (unsigned)rank, (where_), (index), 0ull), false))
#else
#define B2_IN_BOUNDS(index, extent, where_) true
#endif

// One template for one-shot / two-shot / ReduceScatter / NVLS; the differences are data:
// shard_mode picks the range this rank reduces, store_all picks who receives the result.
template <typename T, typename Op, int N, template <class> class PackT, bool kNvls, typename ParamT>
__global__ void __launch_bounds__(kBlockThreads)
reduce_kernel(const __grid_constant__ ParamT param) {
    using P = PackT<T>;
    using Raw = typename P::Raw;
    constexpr int kElems = P::kElems;
    constexpr int NN = N > 0 ? N : kMaxRanks;
    // For the multimem variant the N slot carries the unroll factor (the rank count is a run-time value there). Emulated ranks
    // take 32 bytes per thread and peer, or 16 from five ranks up where those are the packs; two ranks 64, for CTAs that loop
    // (8 MiB in 2 CTAs each 99.8 -> 89.0 us; without a cap 5.6 us either way).
    constexpr int kU = kNvls ? (N > 0 ? N : 4) : (kAllRanksHere<ParamT> ? ((P::kBytes == 16 && N <= 4) || N == 2 ? 2 : 1) : UnrollFor<N, P::kBytes>::value);

    const CollArgs& a = select_args(param);
    const int n = (N > 0 && !kNvls) ? N : a.nranks;
    begin_call<ParamT>((a.shard_mode == kShardSplit ? a.len / n : a.len) * P::kBytes);

    const int rank = kAllRanksHere<ParamT> ? (int)blockIdx.y : a.rank;
    ControlBlock* own = kAllRanksHere<ParamT> ? nullptr : a.ctrl[rank];
    u64 epoch = read_epoch<ParamT>(own);

    const u64 stripe = (u64)gridDim.x * blockDim.x;
    const u64 first = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const int mode = a.shard_mode;
    const int nshards = mode == kShardWhole ? 1 : n;
    const int mine = mode == kShardWhole ? 0 : rank;
    auto shard_lo = [&](int s) -> u64 { return mode == kShardSplit ? (a.len * (u64)s) / (u64)n : 0; };
    auto shard_len = [&](int s) -> u64 {
        return mode == kShardSplit ? (a.len * (u64)(s + 1)) / (u64)n - (a.len * (u64)s) / (u64)n : a.len;
    };

    // 1. Staged input: this CTA copies exactly the packs that the same-numbered CTA of each
    //    peer will read, so the per-CTA barrier below is all the ordering that is needed.
    if (a.user_in != nullptr) {
        void* stage = const_cast<void*>(a.in[rank]);
        for (int s = 0; s < nshards; ++s) {
            const u64 lo = shard_lo(s), len = shard_len(s);
            const u64 dst0 = lo + (u64)s * a.in_stride, src0 = lo + (u64)s * a.uin_stride;
            copy_stripes<P, true>(stage, dst0, a.user_in, src0, first, len, stripe);
        }
    }

    // 2. Every rank's input is ready (and every rank's previous use of `out` is over).
    if (!meet<ParamT>(a, rank, n, epoch, 1u, a.plan_hash)) return;

    // 3. Reduce the own shard.
    {
        const u64 lo = shard_lo(mine), len = shard_len(mine);
        const u64 in0 = lo + (u64)mine * a.in_stride;
        const u64 out0 = mode == kShardBlocks ? 0 : lo;
        const bool scaled = a.scale != 1.0f;
        if constexpr (kNvls) {
            const uint4* mc_in = static_cast<const uint4*>(a.mc_in) + in0;
            uint4* mc_out = static_cast<uint4*>(a.mc_out) + out0;
            for (u64 j = first; j < len; j += stripe * kU) {
                uint4 r[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const u64 jj = j + (u64)u * stripe;
                    if (jj < len) r[u] = multimem_ld_reduce_add<T>(mc_in + jj);
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const u64 jj = j + (u64)u * stripe;
                    if (jj < len) {
                        uint4 v = r[u];
                        if (scaled) {
                            float f[kElems];
                            P::unpack(v, f);
#pragma unroll
                            for (int e = 0; e < kElems; ++e) f[e] *= a.scale;
                            v = P::pack(f);
                        }
                        if (a.store_all) multimem_st16(mc_out + jj, v);
                        else P::store(a.out[rank], out0 + jj, v);
                    }
                }
            }
        } else {
            for (u64 j = first; j < len; j += stripe * kU) {
                Raw r[kU][NN];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const u64 jj = j + (u64)u * stripe;
                    if (jj < len && B2_IN_BOUNDS(in0 + jj, a.in_extent, 30u)) {
#pragma unroll
                        for (int p = 0; p < NN; ++p)
                            if (p < n) r[u][p] = P::load(a.in[p], in0 + jj);
                    }
                }
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const u64 jj = j + (u64)u * stripe;
                    if (jj < len && B2_IN_BOUNDS(in0 + jj, a.in_extent, 30u) && B2_IN_BOUNDS(out0 + jj, a.out_extent, 31u)) {
                        // Fixed order 0..n-1: every rank computes bit-identical results.
                        float acc[kElems];
                        P::unpack(r[u][0], acc);
#pragma unroll
                        for (int p = 1; p < NN; ++p) {
                            if (p < n) {
                                float f[kElems];
                                P::unpack(r[u][p], f);
#pragma unroll
                                for (int e = 0; e < kElems; ++e) acc[e] = Op::apply(acc[e], f[e]);
                            }
                        }
                        if (scaled) {
#pragma unroll
                            for (int e = 0; e < kElems; ++e) acc[e] *= a.scale;
                        }
                        const Raw v = P::pack(acc);
                        if (a.store_all) {
#pragma unroll
                            for (int k = 0; k < NN; ++k) {
                                if (k < n) {
                                    int q = rank + k;  // start with the own copy, then spread over peers
                                    if (q >= n) q -= n;
                                    P::store(a.out[q], out0 + jj, v);
                                }
                            }
                        } else {
                            P::store(a.out[rank], out0 + jj, v);
                        }
                    }
                }
            }
        }
    }

    // 3b. The elements of a ragged or misaligned message that fill no pack, one per thread of CTA 0, in the last rank's shard.
    if constexpr (!kNvls) {
        const unsigned ends = a.head + a.tail;  // at most 15 + 15 (2-byte elements, 32-byte packs): a CTA has 32 threads at least
        if (ends != 0 && blockIdx.x == 0 && threadIdx.x < ends && (mode == kShardWhole || rank == n - 1)) {
            const u64 e = threadIdx.x < a.head ? threadIdx.x : a.len * kElems + threadIdx.x;
            auto first = [&](const void* base) { return static_cast<const T*>(base) - a.head; };
            float acc = Elem<T>::to_f(Narrow<T>::load(first(a.in[0]), e));
            for (int p = 1; p < n; ++p) acc = Op::apply(acc, Elem<T>::to_f(Narrow<T>::load(first(a.in[p]), e)));
            if (a.scale != 1.0f) acc *= a.scale;
            const T v = Elem<T>::from_f(acc);
            if (a.store_all)
                for (int q = 0; q < n; ++q) const_cast<T*>(first(a.out[q]))[e] = v;
            else const_cast<T*>(first(a.out[rank]))[e] = v;
        }
    }

    // 4. Every rank has finished reading inputs and its stores to peers are visible.
    if (!meet<ParamT>(a, rank, n, epoch, 2u, 0ull)) return;

    // 5. Staged output: copy what the same-numbered CTAs of all ranks stored into the arena.
    if (a.user_out != nullptr) {
        for (int s = 0; s < nshards; ++s) {
            const u64 lo = shard_lo(s), len = shard_len(s);
            copy_stripes<P, false>(a.user_out, lo, a.out[rank], lo, first, len, stripe);
        }
    }
    if (!kAllRanksHere<ParamT> && threadIdx.x == 0) own->epoch[blockIdx.x] = epoch;
}

// AllGather: bytes only. push: store the own block into every rank's output; pull: load every
// rank's block into the own output; nvls: one multimem.st per pack reaches every rank.
template <typename RawT, typename ParamT>
__global__ void __launch_bounds__(kBlockThreads)
gather_kernel(const __grid_constant__ ParamT param) {
    const GatherArgs& a = select_args(param);
    begin_call<ParamT>(a.len * sizeof(RawT));
    const int n = a.nranks, rank = kAllRanksHere<ParamT> ? (int)blockIdx.y : a.rank;
    ControlBlock* own = kAllRanksHere<ParamT> ? nullptr : a.ctrl[rank];
    u64 epoch = read_epoch<ParamT>(own);
    const u64 stripe = (u64)gridDim.x * blockDim.x;
    const u64 first = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    constexpr bool kWide = sizeof(RawT) == 16;
    auto load = [](const void* base, u64 i) -> RawT {
        if constexpr (kWide) return ld16_stream(static_cast<const uint4*>(base) + i);
        else return *(static_cast<const volatile RawT*>(base) + i);
    };
    auto store = [](void* base, u64 i, RawT v) {
        if constexpr (kWide) st16(static_cast<uint4*>(base) + i, v);
        else static_cast<RawT*>(base)[i] = v;
    };

    if (a.mode == 1 && a.user_in != nullptr) {
        void* stage = const_cast<void*>(a.in[rank]);
        for (u64 j = first; j < a.len; j += stripe) store(stage, j, load(a.user_in, j));
    }
    if (!meet<ParamT>(a, rank, n, epoch, 1u, a.plan_hash)) return;

    if (a.mode == 0) {
        const u64 base = (u64)rank * a.out_stride;
        for (u64 j = first; j < a.len; j += stripe * 2) {
            const u64 j1 = j + stripe;
            RawT v0 = load(a.in[rank], j), v1;
            if (j1 < a.len) v1 = load(a.in[rank], j1);
            for (int k = 0; k < n; ++k) {
                int q = rank + k;
                if (q >= n) q -= n;
                store(a.out[q], base + j, v0);
                if (j1 < a.len) store(a.out[q], base + j1, v1);
            }
        }
    } else if (a.mode == 1) {
        for (int k = 0; k < n; ++k) {
            int p = rank + k;
            if (p >= n) p -= n;
            const u64 base = (u64)p * a.out_stride;
            for (u64 j = first; j < a.len; j += stripe * 4) {
                RawT v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (j + u * stripe < a.len) v[u] = load(a.in[p], j + u * stripe);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (j + u * stripe < a.len) store(a.out[rank], base + j + u * stripe, v[u]);
            }
        }
    } else {
        if constexpr (kWide) {
            uint4* mc = static_cast<uint4*>(a.mc_out) + (u64)rank * a.out_stride;
            for (u64 j = first; j < a.len; j += stripe) multimem_st16(mc + j, load(a.in[rank], j));
        }
    }

    if (!meet<ParamT>(a, rank, n, epoch, 2u, 0ull)) return;
    if (!kAllRanksHere<ParamT> && threadIdx.x == 0) own->epoch[blockIdx.x] = epoch;
}

// ---- launch helpers ------------------------------------------------------------------------

template <typename A>
using EmulatedRanks = std::conditional_t<kRanksShareGpu, OneGpu<A>, LoopPack<A>>;

// Nothing is staged on one GPU.
template <typename A>
bool fill(OneGpu<A>& all, const A* args, int) {
    all.a = args[0];
    return args[0].user_in == nullptr;
}
template <typename A>
bool fill(LoopPack<A>& all, const A* args, int ranks) {
    for (int r = 0; r < ranks; ++r) all.r[r] = args[r];
    return true;
}

template <typename ParamT>
cudaError_t launch(void (*kernel)(ParamT), const ParamT& param, const LaunchConfig& cfg) {
    dim3 grid(cfg.grid, cfg.loop_ranks > 0 ? cfg.loop_ranks : 1, 1);
    dim3 block(cfg.block, 1, 1);
    if constexpr (kAllRanksHere<ParamT>) {
        cudaLaunchAttribute attrs[1];
        attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[0].val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t config = {};
        config.gridDim = grid;
        config.blockDim = block;
        config.stream = cfg.stream;
        config.attrs = attrs;
        config.numAttrs = 1;
        return cudaLaunchKernelEx(&config, kernel, param);
    } else if (cfg.loop_ranks > 0) {
        // Emulated ranks that wait for one another over flags: all CTAs must be resident, which a cooperative launch checks.
        void* params[] = {const_cast<ParamT*>(&param)};
        return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), grid, block, params, 0,
                                           cfg.stream);
    }
    kernel<<<grid, block, 0, cfg.stream>>>(param);
    return cudaGetLastError();
}

template <typename T, typename Op, template <class> class PackT, bool kNvls, typename ParamT>
cudaError_t launch_reduce_n(int nranks, const ParamT& param, const LaunchConfig& cfg) {
    if constexpr (kNvls) {
        if (cfg.nvls_unroll >= 8) return launch(reduce_kernel<T, Op, 8, PackT, true, ParamT>, param, cfg);
        if (cfg.nvls_unroll <= 1) return launch(reduce_kernel<T, Op, 1, PackT, true, ParamT>, param, cfg);
        if (cfg.nvls_unroll <= 2) return launch(reduce_kernel<T, Op, 2, PackT, true, ParamT>, param, cfg);
        return launch(reduce_kernel<T, Op, 4, PackT, true, ParamT>, param, cfg);
    } else if constexpr (PackT<T>::kBytes < 16) {
        return launch(reduce_kernel<T, Op, 0, PackT, false, ParamT>, param, cfg);
    } else {
        if constexpr (kAllRanksHere<ParamT>) {
            switch (nranks) {
                case 3: return launch(reduce_kernel<T, Op, 3, PackT, false, ParamT>, param, cfg);
                case 5: return launch(reduce_kernel<T, Op, 5, PackT, false, ParamT>, param, cfg);
                case 6: return launch(reduce_kernel<T, Op, 6, PackT, false, ParamT>, param, cfg);
                case 7: return launch(reduce_kernel<T, Op, 7, PackT, false, ParamT>, param, cfg);
                default: break;
            }
        }
        switch (nranks) {
            case 2: return launch(reduce_kernel<T, Op, 2, PackT, false, ParamT>, param, cfg);
            case 4: return launch(reduce_kernel<T, Op, 4, PackT, false, ParamT>, param, cfg);
            case 8: return launch(reduce_kernel<T, Op, 8, PackT, false, ParamT>, param, cfg);
            default:
                if constexpr (kAllRanksHere<ParamT>) return cudaErrorInvalidValue;
                else return launch(reduce_kernel<T, Op, 0, PackT, false, ParamT>, param, cfg);
        }
    }
}

template <typename T, template <class> class PackT, typename ParamT>
cudaError_t launch_reduce_op(RedOp op, int nranks, const ParamT& param, const LaunchConfig& cfg) {
    switch (op) {
        case RedOp::Sum:
        case RedOp::Avg: return launch_reduce_n<T, OpAdd, PackT, false>(nranks, param, cfg);
        case RedOp::Max: return launch_reduce_n<T, OpMax, PackT, false>(nranks, param, cfg);
        case RedOp::Min: return launch_reduce_n<T, OpMin, PackT, false>(nranks, param, cfg);
    }
    return cudaErrorInvalidValue;
}

template <typename T, typename ParamT>
cudaError_t launch_reduce_pack(RedOp op, int pack_bytes, int n, const ParamT& param, const LaunchConfig& cfg) {
    if (pack_bytes == 32) return launch_reduce_op<T, Wide32>(op, n, param, cfg);
    if (pack_bytes == 16) return launch_reduce_op<T, Wide>(op, n, param, cfg);
    return launch_reduce_op<T, Narrow>(op, n, param, cfg);
}

template <typename T>
cudaError_t launch_reduce_t(RedOp op, int pack_bytes, bool nvls, const CollArgs* args, const LaunchConfig& cfg) {
    const int n = args[0].nranks;
    if (cfg.loop_ranks > 0) {
        if (nvls || cfg.loop_ranks > kMaxRanks) return cudaErrorInvalidValue;
        EmulatedRanks<CollArgs> all;
        if (!fill(all, args, cfg.loop_ranks)) return cudaErrorInvalidValue;
        return launch_reduce_pack<T>(op, pack_bytes, n, all, cfg);
    }
    if (nvls) {
        if (pack_bytes != 16 || (op != RedOp::Sum && op != RedOp::Avg)) return cudaErrorInvalidValue;
        return launch_reduce_n<T, OpAdd, Wide, true>(n, args[0], cfg);
    }
    return launch_reduce_pack<T>(op, pack_bytes, n, args[0], cfg);
}

template <typename RawT>
cudaError_t launch_gather_t(const GatherArgs* args, const LaunchConfig& cfg) {
    if (cfg.loop_ranks > 0) {
        if (cfg.loop_ranks > kMaxRanks) return cudaErrorInvalidValue;
        EmulatedRanks<GatherArgs> all;
        if (!fill(all, args, cfg.loop_ranks)) return cudaErrorInvalidValue;
        return launch(gather_kernel<RawT, EmulatedRanks<GatherArgs>>, all, cfg);
    }
    return launch(gather_kernel<RawT, GatherArgs>, args[0], cfg);
}

}  // namespace

cudaError_t launch_reduce(DType dtype, RedOp op, int pack_bytes, bool nvls, const CollArgs* args,
                          const LaunchConfig& cfg) {
    if (pack_bytes != 32 && pack_bytes != 16 && pack_bytes != static_cast<int>(dtype_size(dtype))) return cudaErrorInvalidValue;
    switch (dtype) {
        case DType::Float: return launch_reduce_t<float>(op, pack_bytes, nvls, args, cfg);
        case DType::Float16: return launch_reduce_t<__half>(op, pack_bytes, nvls, args, cfg);
        case DType::BFloat16: return launch_reduce_t<__nv_bfloat16>(op, pack_bytes, nvls, args, cfg);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_gather(const GatherArgs* args, const LaunchConfig& cfg) {
    if (args[0].mode == 2 && (args[0].pack_bytes != 16 || cfg.loop_ranks > 0)) return cudaErrorInvalidValue;
    switch (args[0].pack_bytes) {
        case 16: return launch_gather_t<uint4>(args, cfg);
        case 4: return launch_gather_t<unsigned int>(args, cfg);
        case 2: return launch_gather_t<unsigned short>(args, cfg);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace b200ccl::kernels
