// Ring collectives over Simple-protocol FIFOs for sm_100a.
//
// One CTA per channel. Data moves in slices through per-edge FIFOs that live in the receiver's
// memory (peer stores over NVLink) or in mapped host memory (SHM, socket and RDMA edges). Flow
// control is two monotonically growing step counters per edge, published with st.release.sys and
// polled with ld.acquire.sys; counters persist from launch to launch.
//
// Emulated ranks over device memory run ring_cluster.cu; this kernel plays them only where the turnaround statistics are
// asked for, where host memory or a network lies between them, and in the checking build.
//
// Bound by the chain of slices: a rank can only work on what its neighbour has posted, so what counts is
// the time from one post to the next. Where all ranks run in one launch over device memory, two groups of eight
// warps take the slices in turn, so that one slice is moved while the other waits for its neighbour, for its loads
// or for its release; shared memory hands the order of the posts from group to group (4 ranks: 64 KiB 37.6 -> 27.6
// us, 16 MiB 65.8 -> 59.6 us). FIFOs in host memory keep one group: there each release waits for the other group's
// writes over PCIe as well (4 ranks, 4 MiB: 724 us, 879 us with two). While a slice is moved there is no barrier (one
// comes before an early credit, see run_slice): every thread keeps kBatch vectors of the FIFO and of the local input in
// flight in registers, and the first batch of the local input is loaded BEFORE the wait for the neighbour. (The local
// input used to be staged by TMA through 32 KiB tiles of shared memory, with three block barriers and four dependent
// FIFO loads per thread and tile.)
//
// Parity: nano-nccl src/kernels/ring_simple_kernel.cuh:1118-1237 (schedule 1170-1230:
// direct_send, recv_reduce_send, recv_reduce_copy_send with the fused avg scale, recv_copy_send,
// direct_recv; credit rule 597-634; empty-slice elision 853-859; persistent steps 1152-1163,
// 1232-1236; abort poll 594-611). Differences: channel count is a run-time value; 16-bit types
// accumulate in fp32; every wait is bounded; ReduceScatter and AllGather schedules exist.
#include "kernels/sm100/ring_simple.h"

#include "kernels/sm100/sync.cuh"
#include "kernels/sm100/vec.cuh"
#include "sched/ring_geometry.h"

namespace b200ccl::kernels {

using namespace b200ccl::dev;

namespace {

using u64 = unsigned long long;

constexpr int kRingThreads = 512;
constexpr int kBatch = 8;  // vectors in flight per thread and source
constexpr unsigned kCreditThread = 64, kPostThread = 96;  // of a group: they publish; threads 0 and 32 poll

enum SliceFlags : unsigned {
    kRecv = 1u,        // take the slice from the incoming FIFO
    kLocal = 2u,       // take (or combine with) the local input
    kSend = 4u,        // forward into the outgoing FIFO
    kCopyOut = 8u,     // write into the local output
    kScale = 16u,      // multiply by args.scale before writing (avg, at the pivot only)
};

__device__ __forceinline__ uint4 ld16_volatile(const uint4* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// What the groups of a CTA share: up to which step each side has been published, and whether a group gave up.
struct Turns {
    u64 posted[2];  // 0: slices sent, 1: credits returned
    unsigned failed;
};

struct ChannelState {
    RingChannel ch;
    Turns* turns;
    int group;
    unsigned tid;      // within the group
    unsigned slices;   // non-empty slices so far, of both groups
    bool one_gpu;  // both neighbours run in this launch: their counters need GPU scope only
    u64 send_step;
    u64 recv_step;
};

template <int kGroups>
__device__ __forceinline__ void group_sync(int group) {
    if constexpr (kGroups == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(kRingThreads / kGroups) : "memory");
}
// Barrier of the group; true when `pred` holds in every thread.
template <int kGroups>
__device__ __forceinline__ bool group_sync_and(int group, bool pred) {
    if constexpr (kGroups == 1) return __syncthreads_and(pred ? 1 : 0) != 0;
    unsigned r;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}\n"
        : "=r"(r) : "r"(pred ? 1u : 0u), "r"(group + 1), "n"(kRingThreads / kGroups) : "memory");
    return r != 0;
}

__device__ __forceinline__ u64 ld_acquire_turn(const u64* p) {
    u64 v;
    asm volatile("ld.acquire.cta.shared::cta.u64 %0, [%1];" : "=l"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
template <int kGroups>
__device__ __forceinline__ void st_release_turn(u64* p, u64 v) {
    if constexpr (kGroups > 1)
        asm volatile("st.release.cta.shared::cta.u64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "l"(v) : "memory");
}

// Waits until every slice before `step` has been published; false when the other group gave up. The group that hands
// over has released its slice before, so this group's release covers both.
template <int kGroups>
__device__ __forceinline__ bool wait_turn(const RingArgs& a, Turns& turns, int side, u64 step) {
    if constexpr (kGroups == 1) return true;
    u64 t0 = 0, waited = 0;
    for (unsigned polls = 0;; ++polls) {
        if (ld_acquire_turn(&turns.posted[side]) >= step) return true;
        if (*static_cast<volatile unsigned*>(&turns.failed) != 0u) return false;
        if ((polls & 0xffffu) == 0xffffu) {  // the other group's own waits end after timeout_ns
            if (t0 == 0) t0 = global_timer_ns();
            else if ((waited = global_timer_ns() - t0) > 2 * a.timeout_ns) break;
        }
    }
    report_failure(a.status, a.own_ctrl, nullptr, 0, kStatusTimeout, (unsigned)a.rank, 12u, step, waited);
    *static_cast<volatile unsigned*>(&turns.failed) = 1u;
    return false;
}

// Waits of the two flow-control threads; the outcome is shared through smem.
template <int kGroups>
__device__ __forceinline__ bool wait_flags(const RingArgs& a, ChannelState& st, unsigned flags, u64& t_wait_recv,
                                           u64& t_wait_send) {
    int ok = 1;
    if ((flags & kRecv) && st.tid == 0) {
        const u64 t0 = st.ch.stats ? global_timer_ns() : 0;
        ok = wait_at_least(st.ch.recv_tail, st.recv_step + ring::kSliceSteps, a.own_ctrl, a.timeout_ns, a.status, nullptr,
                           0, (unsigned)((a.rank + a.nranks - 1) % a.nranks), 10u, st.ch.abort_word) ? 1 : 0;
        if (ok && st.ch.abort_word && ld_volatile_u32(st.ch.abort_word) != 0u) ok = 0;
        if (st.ch.stats) t_wait_recv += global_timer_ns() - t0;
    }
    if ((flags & kSend) && st.tid == 32) {
        const u64 t0 = st.ch.stats ? global_timer_ns() : 0;
        // credit: head + kFifoSteps >= step + kSliceSteps
        const u64 want = st.send_step + ring::kSliceSteps >= (u64)ring::kFifoSteps
                             ? st.send_step + ring::kSliceSteps - ring::kFifoSteps : 0;
        ok = wait_at_least(st.ch.send_head, want, a.own_ctrl, a.timeout_ns, a.status, nullptr, 0,
                           (unsigned)((a.rank + 1) % a.nranks), 11u, st.ch.abort_word) ? 1 : 0;
        if (ok && st.ch.abort_word && ld_volatile_u32(st.ch.abort_word) != 0u) ok = 0;
        if (st.ch.stats) t_wait_send += global_timer_ns() - t0;
    }
    if constexpr (kGroups > 1) {
        if (*static_cast<volatile unsigned*>(&st.turns->failed) != 0u) ok = 0;
        if (!ok) *static_cast<volatile unsigned*>(&st.turns->failed) = 1u;
    }
    return group_sync_and<kGroups>(st.group, ok != 0);
}

// One slice: wait, move/combine `n` elements, publish. Returns false when a wait gave up.
template <typename T, typename Op, bool kWide, int kGroups>
__device__ bool run_slice(const RingArgs& a, ChannelState& st, unsigned flags, const T* local_in, T* local_out, u64 n) {
    constexpr int kGroupThreads = kRingThreads / kGroups;
    if (n == 0) {  // empty slice: neither side waits, posts or advances
        if (st.ch.stats && st.tid == 0) atomicAdd(&st.ch.stats->empty_slices, 1ull);
        return true;
    }
    if (kGroups > 1 && (int)(st.slices++ % kGroups) != st.group) {  // the other group's
        if (flags & kRecv) st.recv_step += ring::kSliceSteps;
        if (flags & kSend) st.send_step += ring::kSliceSteps;
        return true;
    }
    const bool recv = flags & kRecv, send = flags & kSend, local = flags & kLocal, copy_out = flags & kCopyOut;
    const bool scaled = (flags & kScale) && a.scale != 1.0f;
    const T* fifo_in = recv ? static_cast<const T*>(st.ch.recv_fifo) + ring::slot_offset(st.recv_step, a.step_elems) : nullptr;
    T* fifo_out = send ? static_cast<T*>(st.ch.send_fifo) + ring::slot_offset(st.send_step, a.step_elems) : nullptr;
    u64 t_wait_recv = 0, t_wait_send = 0, t0 = 0;
    // Small received slices (one 16-byte vector per thread at most) return their FIFO slot to the
    // sender BEFORE they are combined and forwarded: the slot is read into registers, the credit is
    // posted, and only then does the slice go on. On host-memory and network edges, where a credit
    // takes microseconds to arrive, this takes the consumer's own work off the sender's critical path.
    // Inside one GPU the credit is there before the sender has used up its four slots, and the extra barrier and
    // release only lengthen the slice (4 ranks, 64 KiB: 35.9 -> 32.2 us without). Two groups run inside one GPU only and
    // so never take this path; their instances keep the branch because the compiler lays out the slice loop worse without
    // it (2 ranks, 16 MiB: 39.1 us with the branch, 41.1 us without; 4 ranks: 58.6 and 59.7 us).
    // Parity: the reference's early-credit path for slices of at most 4096 bytes
    // (src/kernels/ring_simple_kernel.cuh:486-583, 912-927).
    bool early = false;
    bool ok = true;
    auto combine_element = [&](u64 i) {
        float acc[1];
        if (recv) {
            Narrow<T>::unpack(Narrow<T>::load(fifo_in, i), acc);
            if (local) acc[0] = Op::apply(Elem<T>::to_f(local_in[i]), acc[0]);
        } else {
            acc[0] = Elem<T>::to_f(local_in[i]);
        }
        if (scaled) acc[0] *= a.scale;
        const T out = Elem<T>::from_f(acc[0]);
        if (copy_out) local_out[i] = out;
        if (send) fifo_out[i] = out;
    };
    if constexpr (kWide) {
        constexpr int kElems = 16 / sizeof(T);
        const u64 nvec = n / kElems;
        const unsigned tail = (unsigned)(n - nvec * kElems);  // only the last slice of a ragged message has any
        const uint4* in_v = reinterpret_cast<const uint4*>(local_in);
        const uint4* fifo_v = reinterpret_cast<const uint4*>(fifo_in);
        uint4 loc[kBatch];
        auto load_local = [&](u64 v0) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                if (v0 + u * kGroupThreads < nvec) loc[u] = ld16_stream(in_v + v0 + u * kGroupThreads);
        };
        if (local) load_local(st.tid);
        ok = wait_flags<kGroups>(a, st, flags, t_wait_recv, t_wait_send);
        if (!ok) return false;
        if (st.ch.stats && st.tid == 0) t0 = global_timer_ns();
        early = recv && !st.one_gpu && nvec <= (u64)kGroupThreads && tail == 0;
        uint4 pre = make_uint4(0, 0, 0, 0);
        if (early) {
            int sink = 0;
            if (st.tid < nvec) {
                pre = ld16_volatile(fifo_v + st.tid);
                sink = (pre.x ^ pre.y ^ pre.z ^ pre.w) == 0x5bd1e995u;  // a use of the value: the barrier below then follows the load's arrival
            }
            // The group's __syncthreads_or(): every thread holds its part of the slot.
            (void)group_sync_and<kGroups>(st.group, sink == 0);
            if (st.tid == kCreditThread && wait_turn<kGroups>(a, *st.turns, 1, st.recv_step)) {
                st_release_sys(st.ch.recv_head, st.recv_step + ring::kSliceSteps);
                st_release_turn<kGroups>(&st.turns->posted[1], st.recv_step + ring::kSliceSteps);
            }
        }
        auto combine_store = [&](u64 v, const uint4& got, const uint4& mine) {
            uint4 out = recv ? got : mine;
            if (recv && (local || scaled)) {
                float acc[kElems], f[kElems];
                Wide<T>::unpack(got, acc);
                if (local) {
                    Wide<T>::unpack(mine, f);
#pragma unroll
                    for (int e = 0; e < kElems; ++e) acc[e] = Op::apply(f[e], acc[e]);
                }
                if (scaled) {
#pragma unroll
                    for (int e = 0; e < kElems; ++e) acc[e] *= a.scale;
                }
                out = Wide<T>::pack(acc);
            }
            if (copy_out) st16(reinterpret_cast<uint4*>(local_out) + v, out);
            if (send) st16(reinterpret_cast<uint4*>(fifo_out) + v, out);
        };
        if (early) {
            if (st.tid < nvec) combine_store(st.tid, pre, loc[0]);
        } else {
            for (u64 v0 = st.tid; v0 < nvec; v0 += kBatch * kGroupThreads) {
                uint4 got[kBatch];
                if (recv) {
#pragma unroll
                    for (int u = 0; u < kBatch; ++u)
                        if (v0 + u * kGroupThreads < nvec) got[u] = ld16_volatile(fifo_v + v0 + u * kGroupThreads);
                }
                if (local && v0 != st.tid) load_local(v0);
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                    if (v0 + u * kGroupThreads < nvec) combine_store(v0 + u * kGroupThreads, got[u], loc[u]);
            }
            if (st.tid < tail) combine_element(nvec * kElems + st.tid);
        }
    } else {
        ok = wait_flags<kGroups>(a, st, flags, t_wait_recv, t_wait_send);
        if (!ok) return false;
        if (st.ch.stats && st.tid == 0) t0 = global_timer_ns();
        // More than one element per thread: in batches as well (all_gather of 8 ranks, 500001 bf16: 229 us one by one, 134
        // us; a few hundred elements are faster one by one).
        if (n <= (u64)kGroupThreads) {
            if (st.tid < n) combine_element(st.tid);
        } else {
            for (u64 i0 = st.tid; i0 < n; i0 += kBatch * kGroupThreads) {
                T got[kBatch], mine[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const u64 i = i0 + u * kGroupThreads;
                    if (recv && i < n) got[u] = Narrow<T>::load(fifo_in, i);
                    if (local && i < n) mine[u] = local_in[i];
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const u64 i = i0 + u * kGroupThreads;
                    if (i >= n) continue;
                    float acc = Elem<T>::to_f(recv ? got[u] : mine[u]);
                    if (recv && local) acc = Op::apply(Elem<T>::to_f(mine[u]), acc);
                    if (scaled) acc *= a.scale;
                    const T out = Elem<T>::from_f(acc);
                    if (copy_out) local_out[i] = out;
                    if (send) fifo_out[i] = out;
                }
            }
        }
    }

    // Publish: all data stores of the group happen-before the counters (its __syncthreads(), then release), slice by
    // slice in order. Two warps that do not poll do it.
    group_sync<kGroups>(st.group);
    u64 t1 = 0;
    if (st.ch.stats && st.tid == 0) t1 = global_timer_ns();
    if (recv) {
        if (!early && st.tid == kCreditThread && wait_turn<kGroups>(a, *st.turns, 1, st.recv_step)) {
            st.one_gpu ? st_release_gpu(st.ch.recv_head, st.recv_step + ring::kSliceSteps)
                       : st_release_sys(st.ch.recv_head, st.recv_step + ring::kSliceSteps);
            st_release_turn<kGroups>(&st.turns->posted[1], st.recv_step + ring::kSliceSteps);
        }
        st.recv_step += ring::kSliceSteps;
    }
    if (send) {
        if (st.tid == kPostThread && wait_turn<kGroups>(a, *st.turns, 0, st.send_step)) {
            if (st.ch.send_sizes) {
                st.ch.send_sizes[st.send_step % ring::kFifoSteps] = (unsigned)(n * sizeof(T));
            }
            st.one_gpu ? st_release_gpu(st.ch.send_tail, st.send_step + ring::kSliceSteps)
                       : st_release_sys(st.ch.send_tail, st.send_step + ring::kSliceSteps);
            st_release_turn<kGroups>(&st.turns->posted[0], st.send_step + ring::kSliceSteps);
        }
        st.send_step += ring::kSliceSteps;
    }
    if (st.ch.stats && st.tid == 0) {
        RingTurnaroundStats* s = st.ch.stats;
        atomicAdd(&s->wait_recv_ns, t_wait_recv);
        atomicAdd(&s->compute_ns, t1 - t0);
        atomicAdd(&s->post_ns, global_timer_ns() - t1);
        atomicAdd(&s->slices, 1ull);
    }
    if (st.ch.stats && st.tid == 32 && t_wait_send) atomicAdd(&st.ch.stats->wait_send_ns, t_wait_send);
    return true;
}

// A chunk travels as kSlicesPerChunk slices.
template <typename T, typename Op, bool kWide, int kGroups>
__device__ __forceinline__ bool run_chunk(const RingArgs& a, ChannelState& st, unsigned flags, const T* local_in,
                                          T* local_out, u64 n) {
    const u64 sl = ring::slice_elems(n, sizeof(T), a.step_elems);
#pragma unroll 1
    for (int s = 0; s < ring::kSlicesPerChunk; ++s) {
        const u64 off = (u64)s * sl;
        const u64 sn = ring::clamp_elems(sl, n, off);
        if (!run_slice<T, Op, kWide, kGroups>(a, st, flags, local_in + off, local_out + off, sn)) return false;
    }
    return true;
}

template <typename T, typename Op, bool kWide, int kGroups, typename ParamT>
__global__ void __launch_bounds__(kRingThreads, kWide ? 1 : 2) ring_kernel(const __grid_constant__ ParamT param) {
    __shared__ Turns turns;
    const RingArgs* ap;
    if constexpr (sizeof(ParamT) == sizeof(RingArgs)) ap = reinterpret_cast<const RingArgs*>(&param);
    else ap = reinterpret_cast<const RingArgs*>(&param) + blockIdx.y;
    const RingArgs& a = *ap;
    const int c = blockIdx.x;
    const int n = a.nranks, r = a.rank;

    ChannelState st;
    st.ch = a.channels[c];
    // Network edges name an abort word: a host thread is at their other end.
    st.one_gpu = kRanksShareGpu && sizeof(ParamT) != sizeof(RingArgs) && st.ch.abort_word == nullptr;
    if (threadIdx.x == 0) {
        turns.posted[0] = *st.ch.send_base;
        turns.posted[1] = *st.ch.recv_base;
        turns.failed = 0u;
    }
    __syncthreads();
    st.turns = &turns;
    st.group = (int)(threadIdx.x / (kRingThreads / kGroups));
    st.tid = threadIdx.x % (kRingThreads / kGroups);
    st.slices = 0;
    st.send_step = turns.posted[0];
    st.recv_step = turns.posted[1];
    __syncthreads();  // every thread has read them before a group moves them on

    const T* in = static_cast<const T*>(a.input);
    T* out = static_cast<T*>(a.output);
    // On the 16-byte path parts are cut in whole vectors so that every offset stays aligned.
    constexpr u64 kVecElems = kWide ? 16 / sizeof(T) : 1;
    ring::Part part = ring::channel_part(a.count / kVecElems, c, a.nchannels);
    part.offset *= kVecElems;
    part.count *= kVecElems;
    if (c == a.nchannels - 1) part.count += a.count % kVecElems;  // the rest of a ragged all_reduce
    bool ok = true;
    auto mod = [n](int v) { return ((v % n) + n) % n; };

    // One schedule for the three collectives, so that the slice code exists once: windows of the part, in each of them
    // `steps` chunks. (Four copies with their flags known at compile time spilled registers; the one copy spills up to 24
    // bytes in the 16-byte instances and 48 to 72 in the element ones, which are held to 64 registers.)
    const bool reduces = a.collective != (int)Collective::AllGather, scatters = a.collective == (int)Collective::ReduceScatter;
    const bool both = reduces && !scatters;  // all_reduce: n chunks per window, reduced on the way round and then passed on
    const u64 cs = both ? ring::all_reduce_chunk_elems(part.count, n, sizeof(T), a.step_elems)
                        : ring::block_chunk_elems(part.count, sizeof(T), a.step_elems);
    const u64 window = both ? cs * (u64)n : cs;
    const int steps = both ? 2 * n - 1 : n;
    for (u64 w0 = 0; ok && cs > 0 && w0 < part.count; w0 += window) {
#pragma unroll 1
        for (int j = 1; ok && j <= steps; ++j) {
            unsigned flags;
            if (reduces) {
                if (j == 1) flags = kLocal | kSend;
                else if (j < n) flags = kRecv | kLocal | kSend;
                else if (scatters) flags = kRecv | kLocal | kCopyOut | kScale;  // own block
                else if (j == n) flags = kRecv | kLocal | kSend | kCopyOut | kScale;  // pivot: final value → output and onwards
                else flags = j < steps ? kRecv | kSend | kCopyOut : kRecv | kCopyOut;
            } else {
                flags = j == 1 ? kLocal | kSend | kCopyOut : (j < n ? kRecv | kSend | kCopyOut : kRecv | kCopyOut);
            }
            const int k = mod(reduces ? r - j : r + 1 - j);  // chunk (all_reduce) or block
            u64 at = w0, in_at, out_at;
            if (both) {
                at += (u64)k * cs;
                in_at = out_at = part.offset + at;
            } else {
                const u64 here = part.offset + w0, block = (u64)k * a.count + here;
                in_at = scatters ? block : here;
                out_at = scatters ? here : block;
            }
            ok = run_chunk<T, Op, kWide, kGroups>(a, st, flags, in + in_at, out + out_at, ring::clamp_elems(cs, part.count, at));
        }
    }

    // Progress persists only when the whole schedule ran (an aborted launch leaves the
    // communicator poisoned, as in the reference, kernel:1186-1188).
    ok = __syncthreads_and(ok && turns.failed == 0u) != 0;
    if (ok && threadIdx.x == 0) {
        *st.ch.send_base = st.send_step;
        *st.ch.recv_base = st.recv_step;
    }
}

template <typename T, typename Op, bool kWide>
cudaError_t launch_ring_t(const RingArgs* args, const RingLaunch& cfg) {
    dim3 grid(args[0].nchannels, cfg.loop_ranks > 0 ? cfg.loop_ranks : 1, 1);
    dim3 block(kRingThreads, 1, 1);
    if (cfg.loop_ranks > 0) {
        if (cfg.loop_ranks > kMaxRanks) return cudaErrorInvalidValue;
        LoopPack<RingArgs> pack;
        for (int i = 0; i < cfg.loop_ranks; ++i) pack.r[i] = args[i];
        void* params[] = {&pack};
        const void* kernel = cfg.device_fifos ? reinterpret_cast<const void*>(ring_kernel<T, Op, kWide, 2, LoopPack<RingArgs>>)
                                              : reinterpret_cast<const void*>(ring_kernel<T, Op, kWide, 1, LoopPack<RingArgs>>);
        return cudaLaunchCooperativeKernel(kernel, grid, block, params, 0, cfg.stream);
    }
    ring_kernel<T, Op, kWide, 1, RingArgs><<<grid, block, 0, cfg.stream>>>(args[0]);
    return cudaGetLastError();
}

template <typename T>
cudaError_t launch_ring_op(RedOp op, const RingArgs* args, const RingLaunch& cfg) {
    const bool wide = args[0].wide != 0;
    switch (op) {
        case RedOp::Sum:
        case RedOp::Avg:
            return wide ? launch_ring_t<T, OpAdd, true>(args, cfg) : launch_ring_t<T, OpAdd, false>(args, cfg);
        case RedOp::Max:
            return wide ? launch_ring_t<T, OpMax, true>(args, cfg) : launch_ring_t<T, OpMax, false>(args, cfg);
        case RedOp::Min:
            return wide ? launch_ring_t<T, OpMin, true>(args, cfg) : launch_ring_t<T, OpMin, false>(args, cfg);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

int ring_block_threads() { return kRingThreads; }

cudaError_t launch_ring(DType dtype, RedOp op, const RingArgs* args, const RingLaunch& cfg) {
    switch (dtype) {
        case DType::Float: return launch_ring_op<float>(op, args, cfg);
        case DType::Float16: return launch_ring_op<__half>(op, args, cfg);
        case DType::BFloat16: return launch_ring_op<__nv_bfloat16>(op, args, cfg);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b200ccl::kernels
