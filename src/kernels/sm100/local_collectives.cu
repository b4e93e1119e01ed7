// AllReduce, ReduceScatter and AllGather of ranks that share one device, in one plain launch.
//
// Bound by HBM: every input byte is read once and every output byte is written once. A thread loads the same
// pack of every rank's input, combines them in rank order in fp32, rounds once and stores the result to every
// output that holds it. Nothing waits for anything inside the kernel, so the launch needs no barrier, no flag
// memory and no cooperative launch, any number of CTAs may run, and it is a programmatic dependent of the
// kernel before it.
//
// Layout of the work: a call is cut into segments that share one set of addresses (all_reduce: one;
// reduce_scatter: one per output block; all_gather: one per input), a segment into tiles of one pack per thread, and
// there is one CTA per tile. CTAs start in order and live for one load and one store phase, which keeps the
// window of addresses in flight narrow and the DRAM on reads, then on writes. Measured against CTAs that stay
// and loop (one or two per SM, interleaved or contiguous, 16- to 256-byte windows per thread, and TMA bulk
// copies through shared memory), float sum: 8 ranks x 64 MiB 157.8 us (6.81 TB/s) against 172.7-181.5 us;
// 2 ranks x 512 MiB 308.8 us (6.96 TB/s) against 322-375 us; one rank, 64 MiB 21.2 us against 22.9 us for a
// TMA bulk-copy kernel with one CTA per SM. At these sizes more packs per thread, or 128 or 512 threads, change less than 1 %;
// small grids and reduce_scatter run 128 threads (start_tiles()). CTAs loop only where the caller caps their number.
//
// Lengths and addresses need no alignment beyond the element's. Packs are cut where the INPUTS are aligned (copies whose
// outputs are aligned differently: where the outputs are, see local_shift_copy_kernel); the elements before the first and after the last pack of a segment are handled one by one by the CTA of its first
// tile. Where the outputs are aligned differently (blocks of a ragged reduce_scatter or all_gather), bytes move
// between neighbouring lanes by shuffle so that loads and stores are aligned vectors all the same.
#include "kernels/sm100/local_collectives.h"

#include "kernels/sm100/dev_types.h"
#include "kernels/sm100/vec.cuh"

#include <algorithm>
#include <cstdint>
#include <type_traits>

namespace b200ccl::kernels {

using namespace b200ccl::dev;

namespace {

using u64 = unsigned long long;

constexpr int kThreads = 256;  // or half of that, see start_tiles()
constexpr u64 kSms = 148;

struct LocalArgs {
    const char* in[kMaxRanks];
    char* out[kMaxRanks];
    u64 count;           // elements of one segment
    unsigned tiles;      // of one segment
    float scale;
    unsigned char segments;
    unsigned char nranks;
    unsigned char outs;  // outputs that a segment writes: all of them, or (1) out[s] only
    unsigned char kind;  // Collective
    unsigned char align;  // 16 or 32: what the inputs' addresses (shifted copies: the outputs') agree on
    // Segment s lies s * count elements into every input (reduce_scatter) or every output (all_gather), which reads in[s] only.
    __device__ __forceinline__ u64 in_step(unsigned elem) const { return kind == (int)Collective::ReduceScatter ? count * elem : 0; }
    __device__ __forceinline__ u64 out_step(unsigned elem) const { return kind == (int)Collective::AllGather ? count * elem : 0; }
    __device__ __forceinline__ const char* first_in(unsigned seg) const { return in[kind == (int)Collective::AllGather ? seg : 0]; }
};
// Launching a kernel takes 1.9-2.0 us of host time when the size of its parameters, modulo 64, lies in (16, 32], and
// 2.2-2.5 us otherwise, at any size from 16 to 2848 bytes (CUDA 12.9, driver 580).
static_assert(sizeof(LocalArgs) % 64 > 16 && sizeof(LocalArgs) % 64 <= 32);

// Bytes in flight per thread and input. A copy from one buffer to one buffer wants more (one rank, 64 MiB: 21.6 us
// against 23.4 us with 32 bytes); one to eight buffers does not (8 ranks, 4 MiB blocks: 49.8 us against 46.7 us).
constexpr int kBytes = 32, kCopyBytes = 128;

// Word j.. of eight words shifted right by `bytes` (0 < bytes < 16, even).
__device__ __forceinline__ uint4 shift_pair(const uint4& a, const uint4& b, unsigned bytes) {
    unsigned w0, w1, w2, w3, w4;
    switch (bytes >> 2) {
        case 0: w0 = a.x; w1 = a.y; w2 = a.z; w3 = a.w; w4 = b.x; break;
        case 1: w0 = a.y; w1 = a.z; w2 = a.w; w3 = b.x; w4 = b.y; break;
        case 2: w0 = a.z; w1 = a.w; w2 = b.x; w3 = b.y; w4 = b.z; break;
        default: w0 = a.w; w1 = b.x; w2 = b.y; w3 = b.z; w4 = b.w; break;
    }
    const unsigned bits = (bytes & 3u) * 8u;
    return make_uint4(__funnelshift_r(w0, w1, bits), __funnelshift_r(w1, w2, bits), __funnelshift_r(w2, w3, bits),
                      __funnelshift_r(w3, w4, bits));
}

template <typename T, typename Op, int N>
__device__ __forceinline__ void reduce_one(const LocalArgs& a, unsigned seg, u64 in_off, u64 out_off, u64 e) {
    T v;
    if constexpr (N == 1) {
        v = Narrow<T>::load(a.first_in(seg) + in_off, e);
    } else {
        float acc = 0.0f;
#pragma unroll
        for (int p = 0; p < (N > 0 ? N : kMaxRanks); ++p) {
            if (N > 0 || p < a.nranks) {
                const float f = Elem<T>::to_f(Narrow<T>::load(a.in[p] + in_off, e));
                acc = p == 0 ? f : Op::apply(acc, f);
            }
        }
        v = Elem<T>::from_f(a.scale != 1.0f ? acc * a.scale : acc);
    }
    for (int q = 0; q < a.outs; ++q) reinterpret_cast<T*>(a.out[a.outs == 1 ? seg : q] + out_off)[e] = v;
}

// kShift false: inputs and outputs are all aligned alike, modulo 32. kShift true: the inputs are aligned alike modulo
// 32 or (align 16) modulo 16, and so are the outputs, but differently.
// kSize: threads of a CTA, 0 where the launch says (copies know it when they are compiled: all_gather, 4 ranks, 1 MiB blocks 4.2 us,
// 4.3 without).
template <typename T, typename Op, int N, bool kShift, int kPerThread, int kSize = 0>
__global__ void __launch_bounds__(kThreads, N <= 2 ? 4 : (N <= 4 ? 3 : 2)) local_kernel(const __grid_constant__ LocalArgs a) {
    using P = Wide32<T>;
    constexpr int kElems = P::kElems, kHalf = kElems / 2;
    constexpr int U = kPerThread / 32;
    static_assert(N > 1 || !kShift);  // copies: local_shift_copy_kernel
    const unsigned threads = kSize != 0 ? kSize : blockDim.x;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool scaled = a.scale != 1.0f;
    for (unsigned t = blockIdx.x; t < a.tiles * a.segments; t += gridDim.x) {
        const unsigned seg = t / a.tiles, tile = t - seg * a.tiles;
        const u64 in_off = seg * a.in_step(sizeof(T)), out_off = seg * a.out_step(sizeof(T));
        const char* src0 = a.first_in(seg) + in_off;
        const unsigned cut = kShift ? a.align : 32u;
        const unsigned skew = (unsigned)(reinterpret_cast<std::uintptr_t>(src0) & (cut - 1u));
        const unsigned before = (cut - skew) & (cut - 1u);  // bytes until the inputs are aligned
        const u64 head = before / sizeof(T) < a.count ? before / sizeof(T) : a.count;
        const u64 packs = (a.count - head) / kElems;
        if (tile == 0) {
            const u64 tail0 = head + packs * kElems;
            for (u64 e = threadIdx.x; e < head + (a.count - tail0); e += threads)
                reduce_one<T, Op, N>(a, seg, in_off, out_off, e < head ? e : tail0 + (e - head));
        }
        const u64 in_body = in_off + before, out_body = out_off + before;
        const u64 i0 = (u64)tile * (threads * U) + threadIdx.x;
        const unsigned lane = threadIdx.x & 31u;
        // Bytes by which the outputs are past the inputs' alignment.
        const unsigned m = kShift ? (unsigned)(reinterpret_cast<std::uintptr_t>(a.out[a.outs == 1 ? seg : 0] + out_body) & 15u) : 0u;
        auto body = [&](int p) { return (N == 1 ? src0 - in_off : a.in[p]) + in_body; };
        Raw32 r[U][N];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const u64 i = i0 + u * threads;
            if (i < packs) {
#pragma unroll
                for (int p = 0; p < N; ++p) r[u][p] = kShift && cut == 16u ? P::load_user(body(p), i) : P::load(body(p), i);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const u64 i = i0 + u * threads;
            Raw32 v = r[u][0];
            if constexpr (N > 1) {
                float acc[kElems];
                P::unpack(r[u][0], acc);
#pragma unroll
                for (int p = 1; p < N; ++p) {
                    float f[kElems];
                    P::unpack(r[u][p], f);
#pragma unroll
                    for (int e = 0; e < kElems; ++e) acc[e] = Op::apply(acc[e], f[e]);
                }
                if (scaled) {
#pragma unroll
                    for (int e = 0; e < kElems; ++e) acc[e] *= a.scale;
                }
                v = P::pack(acc);
            }
            if constexpr (!kShift) {
                if (i < packs)
                    for (int q = 0; q < a.outs; ++q) P::store(a.out[a.outs == 1 ? seg : q] + out_body, i, v);
            } else if (m == 0) {
                if (i < packs)
                    for (int q = 0; q < a.outs; ++q) P::store_user(a.out[a.outs == 1 ? seg : q] + out_body, i, v);
            } else {
                // The aligned vectors start s bytes into each half of the lane's pack; the second one ends m bytes into the
                // next lane's pack. The two ends of the warp are stored element by element. (With 16-byte packs, twice the
                // shuffles and ends: reduce_scatter, 3 ranks, 22 MB blocks of odd length 51.0 us, now 42.0; aligned 40.1.)
                const unsigned s = 16u - m;
                uint4 next;
                next.x = __shfl_down_sync(0xffffffffu, v.lo.x, 1);
                next.y = __shfl_down_sync(0xffffffffu, v.lo.y, 1);
                next.z = __shfl_down_sync(0xffffffffu, v.lo.z, 1);
                next.w = __shfl_down_sync(0xffffffffu, v.lo.w, 1);
                if (i < packs) {
                    const bool first = lane == 0u, last = lane == 31u || i + 1 >= packs;
                    const uint4 w0 = shift_pair(v.lo, v.hi, s), w1 = shift_pair(v.hi, next, s);
                    T ends[kElems];
                    *reinterpret_cast<uint4*>(ends) = v.lo;
                    *reinterpret_cast<uint4*>(ends + kHalf) = v.hi;
                    for (int q = 0; q < a.outs; ++q) {
                        char* dst = a.out[a.outs == 1 ? seg : q] + out_body + i * 32ull;
                        st16(reinterpret_cast<uint4*>(dst + s), w0);
                        if (!last) st16(reinterpret_cast<uint4*>(dst + 16 + s), w1);
                        if (first) {
#pragma unroll
                            for (int e = 0; e < kHalf; ++e)
                                if (e * sizeof(T) < s) reinterpret_cast<T*>(dst)[e] = ends[e];
                        }
                        if (last) {
#pragma unroll
                            for (int e = 0; e < kHalf; ++e)
                                if (e * sizeof(T) >= s) reinterpret_cast<T*>(dst + 16)[e] = ends[kHalf + e];
                        }
                    }
                }
            }
        }
    }
}

// Copies whose outputs are aligned differently from their inputs. Stores are most of the traffic of an all_gather, so packs
// of 32 bytes are cut where the OUTPUTS are aligned and the shift is on the loads: every store is a whole sector. (Cut at the
// inputs, neighbouring warps shared sectors, which L2 had to merge. all_gather, bf16, blocks of odd length, us: 8 ranks, 100 KB 6.9
// -> 3.0, 4.2 MB 52.2 -> 48.4, 12 MB 143.7 -> 137.2; 4 ranks, 4.2 MB 15.7 -> 14.7; aligned blocks of 4.2 MB 47.0 and 14.4.) A pack's
// bytes begin `skew` bytes into an aligned vector of the input; the third vector that it touches is the next lane's first.
template <typename T>
__global__ void __launch_bounds__(kThreads, 4) local_shift_copy_kernel(const __grid_constant__ LocalArgs a) {
    constexpr u64 kPack = 32;
    const unsigned threads = blockDim.x;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (unsigned t = blockIdx.x; t < a.tiles * a.segments; t += gridDim.x) {
        const unsigned seg = t / a.tiles, tile = t - seg * a.tiles;
        const u64 out_off = seg * a.out_step(sizeof(T)), bytes = a.count * sizeof(T);
        const char* src0 = a.first_in(seg);
        const unsigned cut = a.align;  // 32 or 16: what the outputs agree on
        u64 before = (cut - (unsigned)(reinterpret_cast<std::uintptr_t>(a.out[0] + out_off) & (cut - 1u))) & (cut - 1u);
        const unsigned skew = (unsigned)(reinterpret_cast<std::uintptr_t>(src0 + before) & 15u);
        if (before < skew) before += cut;  // the first vector lies within the input
        u64 packs = bytes > before ? (bytes - before) / kPack : 0;
        if (skew != 0 && packs != 0 && before - skew + packs * kPack + 16 > bytes) --packs;  // and so does the last
        const u64 head = (before < bytes ? before : bytes) / sizeof(T), tail0 = head + packs * (kPack / sizeof(T));
        if (tile == 0)
            for (u64 e = threadIdx.x; e < head + (a.count - tail0); e += threads)
                reduce_one<T, OpAdd, 1>(a, seg, 0, out_off, e < head ? e : tail0 + (e - head));
        const uint4* src = reinterpret_cast<const uint4*>(src0 + before - skew);
        const u64 i = (u64)tile * threads + threadIdx.x;
        const unsigned lane = threadIdx.x & 31u;
        uint4 w0 = make_uint4(0, 0, 0, 0), w1 = w0, w2;
        Raw32 v;
        if (i < packs) {
            w0 = ld16_stream(src + 2 * i);
            w1 = ld16_stream(src + 2 * i + 1);
        }
        if (skew != 0) {
            uint4 beyond = make_uint4(0, 0, 0, 0);
            const bool last = lane == 31u || i + 1 >= packs;
            if (i < packs && last) beyond = ld16_stream(src + 2 * i + 2);
            w2.x = __shfl_down_sync(0xffffffffu, w0.x, 1);
            w2.y = __shfl_down_sync(0xffffffffu, w0.y, 1);
            w2.z = __shfl_down_sync(0xffffffffu, w0.z, 1);
            w2.w = __shfl_down_sync(0xffffffffu, w0.w, 1);
            if (last) w2 = beyond;
            v.lo = shift_pair(w0, w1, skew);
            v.hi = shift_pair(w1, w2, skew);
        } else {
            v.lo = w0;
            v.hi = w1;
        }
        if (i >= packs) continue;
        for (int q = 0; q < a.outs; ++q) {
            char* dst = a.out[q] + out_off + before + i * kPack;
            if (cut == 32u) {
                st32(dst, v);
            } else {
                st16(reinterpret_cast<uint4*>(dst), v.lo);
                st16(reinterpret_cast<uint4*>(dst) + 1, v.hi);
            }
        }
    }
}

// Inputs (or outputs) that are not aligned alike among themselves: one element per access.
template <typename T, typename Op>
__global__ void __launch_bounds__(kThreads) local_scalar_kernel(const __grid_constant__ LocalArgs a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (unsigned seg = 0; seg < a.segments; ++seg) {
        const u64 in_off = seg * a.in_step(sizeof(T)), out_off = seg * a.out_step(sizeof(T));
        for (u64 e = (u64)blockIdx.x * kThreads + threadIdx.x; e < a.count; e += (u64)gridDim.x * kThreads) {
            if (a.nranks == 1 || a.kind == (int)Collective::AllGather) reduce_one<T, Op, 1>(a, seg, in_off, out_off, e);
            else reduce_one<T, Op, 0>(a, seg, in_off, out_off, e);
        }
    }
}

struct Plan {
    LocalArgs args;
    enum { kElements, kAlike, kShifted } how = kElements;
    int max_ctas = 0;  // 0: one CTA per tile
    int threads = kThreads;
    cudaStream_t stream = nullptr;
};

cudaError_t start(void (*kernel)(LocalArgs), const Plan& p, u64 work, int elem_bytes, LocalLaunch* made) {
    const u64 grid = p.max_ctas > 0 ? std::min<u64>(work, (u64)p.max_ctas) : work;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)grid, 1, 1);
    config.blockDim = dim3(p.threads, 1, 1);
    config.stream = p.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = 1;
    made->grid = (int)grid;
    made->block = p.threads;
    made->pack_bytes = p.how == Plan::kElements ? elem_bytes : 32;
    return cudaLaunchKernelEx(&config, kernel, p.args);
}

// half: the instance for half as many threads, where that is another one.
template <typename T, int kPerThread = kBytes>
cudaError_t start_tiles(void (*kernel)(LocalArgs), Plan& p, LocalLaunch* made, void (*half)(LocalArgs) = nullptr) {
    // Half as many threads where a grid of kThreads leaves SMs idle or with one CTA beside two: an SM stores no faster than its
    // L1 passes on (us, 256 -> 128 threads: all_reduce, 8 ranks, 512 KiB 4.4 -> 3.0, 1 MiB 4.8 -> 4.3, 2 MiB, 256 CTAs, 6.1 -> 6.2; 6 ranks, 1 MiB
    // 3.8 -> 3.2; one rank, 4 MiB 3.6 -> 2.6; all_gather, 8 ranks, blocks of 200 KB 6.1 -> 3.8, of 512 KiB, 512 CTAs, 7.4 -> 7.5). And in
    // a reduce_scatter, which loads most of what it moves (4 ranks, 1 MiB blocks 4.0 -> 3.4; 8 ranks, 2 MiB 23.5 -> 23.3).
    // Not where the caller caps the CTAs below that number: those that there are then loop, and half of them would be missing.
    const bool scatters = p.args.kind == (int)Collective::ReduceScatter;
    const auto tiles_of = [&](int threads) { const u64 tile = (u64)threads * (kPerThread / sizeof(T)); return (p.args.count + tile - 1) / tile; };
    const bool capped = p.max_ctas > 0 && tiles_of(kThreads / 2) * p.args.segments > (u64)p.max_ctas;
    if (!capped && (2 * tiles_of(kThreads) * p.args.segments < 3 * kSms || (scatters && p.args.nranks >= 4))) p.threads = kThreads / 2;
    const u64 tiles = tiles_of(p.threads);
    if (tiles * p.args.segments > 0x7fffffffull) return cudaErrorInvalidValue;
    p.args.tiles = (unsigned)tiles;
    return start(p.threads != kThreads && half != nullptr ? half : kernel, p, tiles * p.args.segments, (int)sizeof(T), made);
}

template <typename T, typename Op>
cudaError_t start_op(Plan& p, LocalLaunch* made) {
    if (p.how == Plan::kElements)
        return start(local_scalar_kernel<T, Op>, p, std::min<u64>((p.args.count + kThreads - 1) / kThreads, 0x7fffffffull), (int)sizeof(T), made);
    switch (p.args.nranks) {
#define B2_LOCAL_N(n) \
    case n: return start_tiles<T>(p.how == Plan::kAlike ? local_kernel<T, Op, n, false, kBytes> : local_kernel<T, Op, n, true, kBytes>, p, made);
        B2_LOCAL_N(2)
        B2_LOCAL_N(3)
        B2_LOCAL_N(4)
        B2_LOCAL_N(5)
        B2_LOCAL_N(6)
        B2_LOCAL_N(7)
        B2_LOCAL_N(8)
#undef B2_LOCAL_N
    }
    return cudaErrorInvalidValue;
}

// Copies: two-byte elements serve every type.
cudaError_t start_copy(Plan& p, LocalLaunch* made) {
    if (p.how == Plan::kAlike && p.args.nranks == 1) return start_tiles<__half, kCopyBytes>(local_kernel<__half, OpAdd, 1, false, kCopyBytes, kThreads>, p, made,
                                                                                                   local_kernel<__half, OpAdd, 1, false, kCopyBytes, kThreads / 2>);
    if (p.how == Plan::kAlike) return start_tiles<__half>(local_kernel<__half, OpAdd, 1, false, kBytes, kThreads>, p, made, local_kernel<__half, OpAdd, 1, false, kBytes, kThreads / 2>);
    if (p.how == Plan::kShifted) {
        const cudaError_t st = start_tiles<__half>(local_shift_copy_kernel<__half>, p, made);
        made->pack_bytes = 16;  // of its loads
        return st;
    }
    return start_op<__half, OpAdd>(p, made);
}

template <typename T>
cudaError_t start_type(RedOp op, Plan& p, LocalLaunch* made) {
    switch (op) {
        case RedOp::Sum:
        case RedOp::Avg: return start_op<T, OpAdd>(p, made);
        case RedOp::Max: return start_op<T, OpMax>(p, made);
        case RedOp::Min: return start_op<T, OpMin>(p, made);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_local(const LocalCall& call, LocalLaunch* made) {
    const int n = call.nranks;
    if (n < 1 || n > kMaxRanks || call.count == 0) return cudaErrorInvalidValue;
    const std::size_t bytes = call.count * dtype_size(call.dtype);
    const bool copies = n == 1 || call.collective == Collective::AllGather;
    Plan p;
    LocalArgs& a = p.args;
    a = LocalArgs{};
    const Collective kind = n == 1 ? Collective::AllReduce : call.collective;  // one rank: the same copy for all three
    a.count = copies ? bytes / 2 : call.count;
    a.nranks = static_cast<unsigned char>(n);
    a.scale = !copies && call.redop == RedOp::Avg ? 1.0f / static_cast<float>(n) : 1.0f;
    a.segments = static_cast<unsigned char>(kind == Collective::AllReduce ? 1 : n);
    a.outs = static_cast<unsigned char>(kind == Collective::ReduceScatter ? 1 : n);
    a.kind = static_cast<unsigned char>(kind);
    // Bits in which the addresses of one side differ, and in which any two addresses of a segment differ.
    std::uintptr_t in_bits = 0, out_bits = 0;
    const auto in0 = reinterpret_cast<std::uintptr_t>(call.in[0]), out0 = reinterpret_cast<std::uintptr_t>(call.out[0]);
    for (int r = 0; r < n; ++r) {
        a.in[r] = static_cast<const char*>(call.in[r]);
        a.out[r] = static_cast<char*>(call.out[r]);
        in_bits |= reinterpret_cast<std::uintptr_t>(call.in[r]) ^ in0;
        out_bits |= reinterpret_cast<std::uintptr_t>(call.out[r]) ^ out0;
    }
    const std::uintptr_t steps = a.segments > 1 ? bytes : 0;
    if (((in_bits | out_bits | (in0 ^ out0) | steps) & 31u) == 0) p.how = Plan::kAlike;
    else if (((in_bits | out_bits) & 15u) == 0) p.how = Plan::kShifted;
    a.align = ((copies ? out_bits : in_bits) & 31u) == 0 ? 32 : 16;
    p.max_ctas = call.max_ctas;
    p.stream = call.stream;
    if (copies) return start_copy(p, made);
    switch (call.dtype) {
        case DType::Float: return start_type<float>(call.redop, p, made);
        case DType::Float16: return start_type<__half>(call.redop, p, made);
        case DType::BFloat16: return start_type<__nv_bfloat16>(call.redop, p, made);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b200ccl::kernels

// ---------------------------------------------------------------------------------------------
// Allocation-free single-GPU all-reduce (declaration and contract: kernels/sm100/no_alloc.h).
// The launch above needs no memory of its own, so there is nothing to add but the checks.

#include "kernels/sm100/no_alloc.h"

#include <string>

namespace b200ccl::kernels {
// Message of the calling thread's last failure, shared with the C interface (b2_last_error).
void set_last_error_message(const std::string& message);
}  // namespace b200ccl::kernels

extern "C" int b2_local_all_reduce_no_alloc(const void* const* inputs, void* const* outputs, int nranks, size_t count,
                                            int dtype, int redop, void* stream, void* /*status_record*/) {
    using namespace b200ccl;
    auto reject = [](const std::string& why) {
        kernels::set_last_error_message("b2_local_all_reduce_no_alloc: " + why);
        return 2;
    };
    if (nranks < 1 || nranks > B2_NO_ALLOC_MAX_RANKS)
        return reject("nranks = " + std::to_string(nranks) + " is outside 1.." + std::to_string(B2_NO_ALLOC_MAX_RANKS));
    if (count == 0) return reject("count must be positive");
    if (dtype < 0 || dtype > 2) return reject("unsupported dtype");
    if (redop < 0 || redop > 3) return reject("unknown reduction operator");
    if (inputs == nullptr || outputs == nullptr) return reject("inputs and outputs must be non-null");
    const std::size_t elem_bytes = dtype_size(static_cast<DType>(dtype));
    if (count > SIZE_MAX / elem_bytes) return reject("count * element size does not fit in size_t");
    const std::size_t span = count * elem_bytes;
    // Byte ranges [ptr, ptr + span) of two buffers share at least one byte.
    auto overlap = [span](const void* a, const void* b) {
        const std::uintptr_t x = reinterpret_cast<std::uintptr_t>(a), y = reinterpret_cast<std::uintptr_t>(b);
        return x < y ? y - x < span : x - y < span;
    };
    for (int r = 0; r < nranks; ++r) {
        if (inputs[r] == nullptr || outputs[r] == nullptr) return reject("every buffer must be non-null");
        if (reinterpret_cast<std::uintptr_t>(inputs[r]) > UINTPTR_MAX - span ||
            reinterpret_cast<std::uintptr_t>(outputs[r]) > UINTPTR_MAX - span)
            return reject("a buffer's byte range wraps around the address space");
    }
    for (int r = 0; r < nranks; ++r) {
        for (int q = 0; q < nranks; ++q) {
            if (inputs[r] == outputs[q]) return reject("in-place operation is not supported");
            if (overlap(inputs[r], outputs[q]))
                return reject("input " + std::to_string(r) + " and output " + std::to_string(q) + " overlap");
            if (q > r && overlap(outputs[r], outputs[q]))
                return reject("outputs " + std::to_string(r) + " and " + std::to_string(q) + " overlap");
        }
    }
    kernels::LocalCall call;
    call.collective = Collective::AllReduce;
    call.dtype = static_cast<DType>(dtype);
    call.redop = static_cast<RedOp>(redop);
    call.nranks = nranks;
    call.in = inputs;
    call.out = outputs;
    call.count = count;
    call.stream = static_cast<cudaStream_t>(stream);
    kernels::LocalLaunch made;
    const cudaError_t st = kernels::launch_local(call, &made);
    if (st != cudaSuccess) {
        kernels::set_last_error_message(std::string("b2_local_all_reduce_no_alloc: launch failed: ") + cudaGetErrorString(st));
        (void)cudaGetLastError();
        return 1;
    }
    return 0;
}
