// Low-latency AllReduce for small messages (up to 128 KiB): no barrier at all. Every rank stores
// each 4-byte word of its input, paired with the number of this call, straight into a slot of
// every rank's receive area (one 8-byte store, which arrives whole). A receiver spins on the slot
// until the call number matches, so the data is its own "ready" flag and the whole exchange costs
// one NVLink crossing instead of the two barrier round-trips of the one-shot kernel. Slots
// alternate between two parities: a rank can be at most one call ahead of a peer (it cannot finish
// a call without that peer's data for it), so a slot is never overwritten while it may still be read.
// Neither input nor output needs to be addressable by peers: only the receive areas are.
//
// The reference has no counterpart (its smallest latency is 2(N-1) ring hops); the idea is the
// flag-in-data "LL" protocol known from NCCL, written here for direct all-to-all exchange.
#include "kernels/sm100/ll_allreduce.h"

#include "kernels/sm100/sync.cuh"
#include "kernels/sm100/vec.cuh"

#include <cstdint>
#include <type_traits>

namespace b200ccl::kernels {

using namespace b200ccl::dev;

namespace {

using u64 = unsigned long long;

__device__ __forceinline__ void st_slot(u64* p, unsigned data, unsigned flag) {
    asm volatile("st.relaxed.sys.global.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(data), "r"(flag) : "memory");
}
__device__ __forceinline__ uint2 ld_slot(const u64* p) {
    uint2 v;
    asm volatile("ld.relaxed.sys.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
    return v;
}

template <typename T>
struct Word;  // one 4-byte word ↔ fp32 lanes
template <>
struct Word<float> {
    static constexpr int kLanes = 1;
    static __device__ __forceinline__ void unpack(unsigned w, float (&f)[1]) { f[0] = __uint_as_float(w); }
    static __device__ __forceinline__ unsigned pack(const float (&f)[1]) { return __float_as_uint(f[0]); }
};
template <>
struct Word<__half> {
    static constexpr int kLanes = 2;
    static __device__ __forceinline__ void unpack(unsigned w, float (&f)[2]) { float2 v = h2_to_f2(w); f[0] = v.x; f[1] = v.y; }
    static __device__ __forceinline__ unsigned pack(const float (&f)[2]) { return f2_to_h2(f[0], f[1]); }
};
template <>
struct Word<__nv_bfloat16> {
    static constexpr int kLanes = 2;
    static __device__ __forceinline__ void unpack(unsigned w, float (&f)[2]) { float2 v = b2_to_f2(w); f[0] = v.x; f[1] = v.y; }
    static __device__ __forceinline__ unsigned pack(const float (&f)[2]) { return f2_to_b2(f[0], f[1]); }
};

constexpr unsigned kWordsAtATime = kLlCtas * kBlockThreads;  // words that the CTAs of a rank take at a time

// Emulated ranks: what they share. The rank is blockIdx.y.
struct LlOneGpuArgs {
    const void* in[kMaxRanks];
    void* out[kMaxRanks];
    u64* area[kMaxRanks];
    ControlBlock* ctrl[kMaxRanks];
    Status* status;
    u64 timeout_ns;
    unsigned nwords;
    float scale;
    int nranks;
    int pad;
};
static_assert(sizeof(LlOneGpuArgs) % 64 > 16 && sizeof(LlOneGpuArgs) % 64 <= 32);  // launches fastest, see local_collectives.cu

// 1. Publish, kBatch words per thread at a time. Between GPUs: word w of this rank goes to slot (parity, rank, w) of every rank.
template <int kBatch>
__device__ __forceinline__ void publish(const LlArgs& a, int rank, u64 parity, unsigned flag, unsigned first) {
    const int n = a.nranks;
    const unsigned* in = static_cast<const unsigned*>(a.in);
    auto has = [&](unsigned w0, int u) { return u == 0 || w0 + u * kWordsAtATime < a.nwords; };  // the loops see to the first one
    for (unsigned w0 = first; w0 < a.nwords; w0 += kWordsAtATime * kBatch) {
        unsigned v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (has(w0, u)) v[u] = in[w0 + u * kWordsAtATime];
        const u64 slot = (parity * (u64)n + (u64)rank) * kLlMaxWords + w0;
        for (int k = 0; k < n; ++k) {
            int q = rank + k;
            if (q >= n) q -= n;
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (has(w0, u)) st_slot(a.area[q] + slot + u * kWordsAtATime, v[u], flag);
        }
    }
}

// Emulated ranks: the thread that will collect a word for this rank stores every rank's word into this rank's slots itself. The
// same stores in all, but a thread only ever waits for its own: no CTA waits for another one, and the launch is a plain
// programmatic dependent of the one before instead of a cooperative one. Not in place: see outputs_overlap_inputs(). (A thread that did so for every rank at once,
// ranks^2 slots, was slower from five ranks up: 8 ranks, 16 KiB 10.1 us.) Cooperative -> now: 2 ranks, 1 KiB 4.3 -> 3.1 us, 128 KiB 10.2 -> 7.2;
// 8 ranks, 1 KiB 4.5 -> 3.3, 16 KiB 6.1 -> 3.4, 64 KiB 8.2 -> 6.7, 128 KiB 14.3 -> 11.4.
template <int kBatch>
__device__ __forceinline__ void publish(const LlOneGpuArgs& a, int rank, u64 parity, unsigned flag, unsigned first) {
    const int n = a.nranks;
    u64* own_area = a.area[rank] + parity * (u64)n * kLlMaxWords;
    auto has = [&](unsigned w0, int u) { return u == 0 || w0 + u * kWordsAtATime < a.nwords; };
    for (unsigned w0 = first; w0 < a.nwords; w0 += kWordsAtATime * kBatch) {
        unsigned v[kBatch][kMaxRanks];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
#pragma unroll
            for (int p = 0; p < kMaxRanks; ++p)
                if (p < n && has(w0, u)) v[u][p] = static_cast<const unsigned*>(a.in[p])[w0 + u * kWordsAtATime];
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
#pragma unroll
            for (int p = 0; p < kMaxRanks; ++p)
                if (p < n && has(w0, u)) st_slot(own_area + (u64)p * kLlMaxWords + w0 + u * kWordsAtATime, v[u][p], flag);
    }
}

template <typename A>
__device__ __forceinline__ unsigned* output(const A& a, int rank) {
    if constexpr (std::is_same_v<A, LlOneGpuArgs>) return static_cast<unsigned*>(a.out[rank]);
    else return static_cast<unsigned*>(a.out);
}

// One rank's part of the exchange; false when a wait gave up.
template <typename T, typename Op, int kBatch, typename A>
__device__ __forceinline__ bool exchange(const A& a, int rank, u64 call) {
    static_assert(kBatch * kMaxRanks <= 32, "pending words are bits of one register");
    const int n = a.nranks;
    const unsigned flag = static_cast<unsigned>(call % 0xffffffffull) + 1u;  // never 0: a zeroed area matches no call
    const u64 parity = call & 1ull;
    unsigned* out = output(a, rank);
    ControlBlock* own = a.ctrl[rank];
    const unsigned first = blockIdx.x * kBlockThreads + threadIdx.x;
    auto has = [&](unsigned w0, int u) { return u == 0 || w0 + u * kWordsAtATime < a.nwords; };

    publish<kBatch>(a, rank, parity, flag, first);
    // 2. Collect: the slots of all sources and of kBatch words are loaded together, then only those whose call number
    //    has not arrived yet are polled again; combine in rank order.
    bool ok = true;
    const u64 t0 = global_timer_ns();
    const u64* own_area = a.area[rank] + parity * (u64)n * kLlMaxWords;
    for (unsigned w0 = first; ok && w0 < a.nwords; w0 += kWordsAtATime * kBatch) {
        uint2 v[kBatch][kMaxRanks];
        unsigned pending = 0u;  // bit u * kMaxRanks + p: word u of rank p
#pragma unroll
        for (int u = 0; u < kBatch; ++u)
            if (has(w0, u)) pending |= ((1u << n) - 1u) << (u * kMaxRanks);
        unsigned polls = 0;
        while (pending != 0u) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
#pragma unroll
                for (int p = 0; p < kMaxRanks; ++p)
                    if (pending & (1u << (u * kMaxRanks + p))) v[u][p] = ld_slot(own_area + (u64)p * kLlMaxWords + w0 + u * kWordsAtATime);
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
#pragma unroll
                for (int p = 0; p < kMaxRanks; ++p)
                    if ((pending & (1u << (u * kMaxRanks + p))) && v[u][p].y == flag) pending &= ~(1u << (u * kMaxRanks + p));
            if (pending != 0u && (++polls & 255u) == 0u) {
                const unsigned who = (unsigned)(__ffs((int)pending) - 1) % kMaxRanks;
                if (ld_volatile_u32(&own->abort_flag) != 0u) {
                    report_failure(a.status, own, nullptr, 0, kStatusAborted, who, 20u, call, global_timer_ns() - t0);
                    ok = false;
                    break;
                }
                const u64 waited = global_timer_ns() - t0;
                if (waited > a.timeout_ns) {
                    report_failure(a.status, own, a.ctrl, n, kStatusTimeout, who, 20u, call, waited);
                    ok = false;
                    break;
                }
            }
        }
        if (!ok) break;
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            if (!has(w0, u)) break;
            float acc[Word<T>::kLanes];
            Word<T>::unpack(v[u][0].x, acc);
#pragma unroll
            for (int p = 1; p < kMaxRanks; ++p) {
                if (p < n) {
                    float f[Word<T>::kLanes];
                    Word<T>::unpack(v[u][p].x, f);
#pragma unroll
                    for (int e = 0; e < Word<T>::kLanes; ++e) acc[e] = Op::apply(acc[e], f[e]);
                }
            }
            if (a.scale != 1.0f) {
#pragma unroll
                for (int e = 0; e < Word<T>::kLanes; ++e) acc[e] *= a.scale;
            }
            out[w0 + u * kWordsAtATime] = Word<T>::pack(acc);
        }
    }
    return ok;
}

template <typename A>
__device__ __forceinline__ const A& select_args(const A& a) { return a; }
template <typename A>
__device__ __forceinline__ const A& select_args(const LoopPack<A>& all) { return all.r[blockIdx.y]; }

template <typename T, typename Op, int kBatch, typename ParamT>
__global__ void __launch_bounds__(kBlockThreads) ll_kernel(const __grid_constant__ ParamT param) {
    constexpr bool kOneGpu = std::is_same_v<ParamT, LlOneGpuArgs>;
    if constexpr (kOneGpu) {
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    const auto& a = select_args(param);
    int rank;
    if constexpr (kOneGpu) rank = (int)blockIdx.y;
    else rank = a.rank;
    // Every thread reads the CTA's call counter; thread 0 writes it back at the end.
    ControlBlock* own = a.ctrl[rank];
    const u64 call = own->ll_epoch[blockIdx.x] + 1;
    const bool ok = exchange<T, Op, kBatch>(a, rank, call);
    // A CTA whose wait gave up leaves its counter alone: the communicator is poisoned anyway.
    if (__syncthreads_and(ok ? 1 : 0) && threadIdx.x == 0) own->ll_epoch[blockIdx.x] = call;
}

// Whether an output overlaps an input, its own rank's (a call in place) or another one's. The thread that writes a word of it knows
// that every rank has read that word only where the ranks wait for one another.
bool outputs_overlap_inputs(const LlArgs* args, int ranks) {
    const std::uintptr_t bytes = 4ull * args[0].nwords;
    for (int q = 0; q < ranks; ++q)
        for (int r = 0; r < ranks; ++r) {
            const auto out = reinterpret_cast<std::uintptr_t>(args[q].out), in = reinterpret_cast<std::uintptr_t>(args[r].in);
            if (out < in + bytes && in < out + bytes) return true;
        }
    return false;
}

template <typename T, typename Op, int kBatch>
cudaError_t launch_ll_t(const LlArgs* args, int loop_ranks, cudaStream_t stream, bool waiting) {
    dim3 grid(kLlCtas, loop_ranks > 0 ? loop_ranks : 1, 1), block(kBlockThreads, 1, 1);
    if (loop_ranks > kMaxRanks) return cudaErrorInvalidValue;
    if (loop_ranks > 0) {
        if (!waiting) {
            LlOneGpuArgs a = {};
            for (int r = 0; r < loop_ranks; ++r) {
                a.in[r] = args[r].in;
                a.out[r] = args[r].out;
                a.area[r] = args[0].area[r];
                a.ctrl[r] = args[0].ctrl[r];
            }
            a.status = args[0].status;
            a.timeout_ns = args[0].timeout_ns;
            a.nwords = args[0].nwords;
            a.scale = args[0].scale;
            a.nranks = loop_ranks;
            cudaLaunchAttribute attrs[1];
            attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attrs[0].val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t config = {};
            config.gridDim = grid;
            config.blockDim = block;
            config.stream = stream;
            config.attrs = attrs;
            config.numAttrs = 1;
            return cudaLaunchKernelEx(&config, ll_kernel<T, Op, kBatch, LlOneGpuArgs>, a);
        }
        // Ranks that wait for one another: all CTAs must be resident, which a cooperative launch checks.
        LoopPack<LlArgs> pack;
        for (int r = 0; r < loop_ranks; ++r) pack.r[r] = args[r];
        void* params[] = {&pack};
        return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(ll_kernel<T, Op, kBatch, LoopPack<LlArgs>>), grid, block, params, 0, stream);
    }
    ll_kernel<T, Op, kBatch, LlArgs><<<grid, block, 0, stream>>>(args[0]);
    return cudaGetLastError();
}

// One word at a time, each takes a round trip to the slots; but a batch that is not full costs its registers (91 or 124 against 40)
// and conditions. Ranks that wait for one another (as emulated ranks did; us, one at a time / four): 20000 bytes, 2 ranks 4.6 / 6.1,
// 8 ranks 6.2 / 6.8; level at 40000 and 70000 bytes; 128 KiB, 8 ranks 14.3 / 12.3. So from four full words up. Emulated ranks as they are
// now: 32 KiB, 2 ranks 3.2 / 4.3, 4 ranks 4.3 / 4.4, 6 ranks 6.3 / 4.7, 8 ranks 7.3 / 5.2; 64 KiB, 2 ranks 4.9 / 4.6, 8 ranks 12.6 / 6.7.
template <typename T, typename Op>
cudaError_t launch_ll_size(const LlArgs* args, int loop_ranks, cudaStream_t stream) {
    const bool waiting = !kRanksShareGpu || loop_ranks == 0 || outputs_overlap_inputs(args, loop_ranks);
    const unsigned singles = waiting ? 4u : (loop_ranks <= 5 ? 2u : 1u);
    return args[0].nwords <= singles * kWordsAtATime ? launch_ll_t<T, Op, 1>(args, loop_ranks, stream, waiting)
                                                     : launch_ll_t<T, Op, 4>(args, loop_ranks, stream, waiting);
}

template <typename T>
cudaError_t launch_ll_op(RedOp op, const LlArgs* args, int loop_ranks, cudaStream_t stream) {
    switch (op) {
        case RedOp::Sum:
        case RedOp::Avg: return launch_ll_size<T, OpAdd>(args, loop_ranks, stream);
        case RedOp::Max: return launch_ll_size<T, OpMax>(args, loop_ranks, stream);
        case RedOp::Min: return launch_ll_size<T, OpMin>(args, loop_ranks, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

std::size_t ll_area_bytes(int nranks) { return std::size_t(2) * nranks * kLlMaxWords * sizeof(unsigned long long); }

cudaError_t launch_ll_all_reduce(DType dtype, RedOp op, const LlArgs* args, int loop_ranks, cudaStream_t stream) {
    switch (dtype) {
        case DType::Float: return launch_ll_op<float>(op, args, loop_ranks, stream);
        case DType::Float16: return launch_ll_op<__half>(op, args, loop_ranks, stream);
        case DType::BFloat16: return launch_ll_op<__nv_bfloat16>(op, args, loop_ranks, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b200ccl::kernels
