// AllReduce, ReduceScatter and AllGather of emulated ranks over host memory, two-shot instead of a ring.
//
// Bound by PCIe. A ring of n ranks sends 2(n-1)/n of the message over every edge, written to host memory by one rank and read
// by the next, in 2(n-1) dependent hops of about 13 us each. Here a rank writes its input for the share of every other rank
// ((n-1)/n of the message), reduces its own share of everybody's input, and writes that once (1/n) for all others to read: the
// reads are the same, the writes half as many for large n, and there are two hops. It also adds in rank order in fp32 and
// rounds once. All_reduce of 4 ranks, us, ring -> here: 4 KiB 97 -> 23, 256 KiB 107 -> 71, 4 MiB 729 -> 704 (25 MB read, 17 written: a copy
// kernel takes 585 for as much); 8 ranks, 4 KiB 265 -> 31, 4 MiB 1681 -> 1472. What is left to the copy goes into the system-scope
// releases and the waits for flags, about 13 us for every tile of a CTA; more reads in flight (8 instead of 4 per thread) or more
// CTAs make it slower. When each is the better one: exchange_pays() in sched/plan.cc.
//
// A tile is a chunk of every rank's share; a CTA takes the tiles cta, cta + ctas, ... and passes every one through three
// steps: give (own input into the others' part slots), reduce (the parts of its own share; the result into its result slot),
// take (the others' results into the output). Tile t is reduced, and t+1 given meanwhile, so that PCIe is busy both ways; then
// t-1 is taken, whose results have had that long to arrive. Slots are used again after three tiles and need no credits: who has
// taken tile t from rank q knows that q has read its part of t; and who gives tile t+3 has taken t. ReduceScatter and
// AllGather run the same steps with nothing in the slots that they do not need.
//
// Every wait is bounded; the launch is cooperative.
#include "kernels/sm100/host_exchange.h"

#include "kernels/sm100/rows.cuh"
#include "kernels/sm100/sync.cuh"
#include "sched/ring_geometry.h"

#include <algorithm>

namespace b200ccl::kernels {

using namespace b200ccl::dev;

namespace {

using u64 = unsigned long long;

constexpr int kThreads = 512, kWarps = kThreads / 32;

__device__ __forceinline__ uint4 ld16_host(const unsigned char* p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

template <typename T, typename Op, bool kWide>
__global__ void __launch_bounds__(kThreads, 1) host_exchange_kernel(const __grid_constant__ HostExchangeArgs a) {
    using R = Row<T, kWide>;
    constexpr int kElems = R::kElems;
    const int n = a.nranks, r = (int)blockIdx.y, cta = (int)blockIdx.x;
    const unsigned warp = threadIdx.x / 32u, lane = threadIdx.x & 31u;
    const bool reduces = a.collective != (int)Collective::AllGather, scatters = a.collective == (int)Collective::ReduceScatter;
    const bool gathers = !scatters, both = reduces && gathers;
    const unsigned lead = kWide ? a.lead : 0u;
    const T* in = static_cast<const T*>(a.in[r]) - lead;
    T* out = static_cast<T*>(a.out[r]) - lead;
    const int ctas = a.ctas;
    u64* own_tiles = a.tiles + (u64)r * ctas + cta;
    const u64 before = *own_tiles;

    const u64 total = a.count + lead;  // elements from the boundary on: of the message (all_reduce) or of a block
    // A tile: `rows` rows of every rank's share, or of every block. In an all_reduce the shares of a tile follow one another.
    struct Tile {
        u64 row0;
        unsigned rows;  // 0: none
    };
    // Where rank q's chunk lies in a buffer of all shares or blocks, in one of a single block, and its elements.
    auto block_at = [&](int q, const Tile& c) { return (both ? (u64)n * c.row0 + (u64)q * c.rows : c.row0) * R::kSize; };
    auto whole_at = [&](int q, const Tile& c) { return both ? block_at(q, c) : (u64)q * a.count + block_at(q, c); };
    auto size_of = [&](int q, const Tile& c) { return (unsigned)ring::clamp_elems(c.rows * R::kSize, total, block_at(q, c)); };
    auto part_slot = [&](int to, int from, u64 t) { return a.parts + ((((u64)to * n + from) * ctas + cta) * kHostSlots + t % kHostSlots) * kHostChunkBytes; };
    auto result_slot = [&](int from, u64 t) { return a.results + (((u64)from * ctas + cta) * kHostSlots + t % kHostSlots) * kHostChunkBytes; };
    auto given = [&](int to, int from) { return a.given + ((u64)to * n + from) * ctas + cta; };
    auto done = [&](int from) { return a.done + (u64)from * ctas + cta; };

    // Waits of the lanes of warp 0 for one peer each.
    auto wait_all = [&](auto flag_of, u64 want, unsigned where) {
        int ok = 1;
        if (threadIdx.x < (unsigned)n && (int)threadIdx.x != r)
            ok = wait_at_least(flag_of((int)threadIdx.x), want, a.ctrl[r], a.timeout_ns, a.status[r], nullptr, 0, threadIdx.x, where) ? 1 : 0;
        return __syncthreads_and(ok) != 0;
    };

    // Row i of own input for the other ranks' shares: read, and written into its slot; t counts tiles over all calls.
    struct Given {
        uint4 v;
        unsigned char* to;  // null: no such element
    };
    auto give_load = [&](unsigned i, const Tile& c, u64 t) {
        Given g{make_uint4(0, 0, 0, 0), nullptr};
        const unsigned row = i % c.rows, e = row * R::kSize + R::first(lane);
        int q = r + 1 + (int)(i / c.rows);
        if (q >= n) q -= n;
        const unsigned size = size_of(q, c);
        if (e < size) {
            g.v = R::load(in, whole_at(q, c), e, size, lead);
            g.to = part_slot(q, r, t) + row * 512u + lane * 16u;
        }
        return g;
    };
    auto give_store = [](const Given& g) {
        if (g.to != nullptr) st16(reinterpret_cast<uint4*>(g.to), g.v);
    };
    // Says that everything up to here is written: parts of `parts` tiles, results of `results` tiles.
    auto publish = [&](u64 parts, u64 results) {
        __syncthreads();
        if (threadIdx.x < (unsigned)n) {
            if ((int)threadIdx.x != r) st_release_sys(given((int)threadIdx.x, r), parts);
            else st_release_sys(done(r), results);
        }
    };

    // Own share of a tile, and the parts of the next tile for the others while its reads are under way.
    auto reduce = [&](const Tile& c, const Tile& next, u64 t) {
        if (!wait_all([&](int p) { return given(r, p); }, t + 1, 60u)) return false;
        const unsigned size = size_of(r, c);
        const u64 in_at = reduces ? whole_at(r, c) : block_at(r, c), out_at = scatters ? block_at(r, c) : whole_at(r, c);
        // Rows of the next tile that go with each row of this one (tiles grow up to twofold).
        const unsigned give_rows = reduces ? (unsigned)(n - 1) * next.rows : 0u;
        unsigned given_rows = warp;
        for (unsigned row = warp; row < c.rows; row += kWarps) {
            const unsigned e = row * R::kSize + R::first(lane);
            const bool mine = e < size;
            uint4 v = make_uint4(0, 0, 0, 0), got[kMaxRanks];
            if (mine && reduces) {
#pragma unroll
                for (int p = 0; p < kMaxRanks; ++p)
                    if (p < n && p != r) got[p] = ld16_host(part_slot(r, p, t) + row * 512u + lane * 16u);
            }
            if (mine) v = R::load(in, in_at, e, size, lead);
            constexpr int kBatch = 4;
            const unsigned until = row + kWarps < c.rows ? min(give_rows, (unsigned)((u64)give_rows * (row / kWarps + 1) * kWarps / c.rows)) : give_rows;
            while (given_rows < until) {
                Given g[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                    if (given_rows + u * kWarps < until) g[u] = give_load(given_rows + u * kWarps, next, t + 1);
#pragma unroll
                for (int u = 0; u < kBatch; ++u)
                    if (given_rows + u * kWarps < until) give_store(g[u]);
                for (int u = 0; u < kBatch && given_rows < until; ++u) given_rows += kWarps;
            }
            if (!mine) continue;
            if (reduces) {
                float acc[kElems], f[kElems];
                Wide<T>::unpack(r == 0 ? v : got[0], acc);
#pragma unroll
                for (int p = 1; p < kMaxRanks; ++p) {
                    if (p >= n) break;
                    Wide<T>::unpack(p == r ? v : got[p], f);
#pragma unroll
                    for (int k = 0; k < kElems; ++k) acc[k] = Op::apply(acc[k], f[k]);
                }
                if (a.scale != 1.0f) {
#pragma unroll
                    for (int k = 0; k < kElems; ++k) acc[k] *= a.scale;
                }
                v = Wide<T>::pack(acc);
            }
            if (gathers) st16(reinterpret_cast<uint4*>(result_slot(r, t) + row * 512u) + lane, v);
            R::store(out, out_at, e, size, lead, v);
        }
        // A warp without a row of its own still has some to give.
        for (; given_rows < give_rows; given_rows += kWarps) give_store(give_load(given_rows, next, t + 1));
        publish(next.rows != 0 ? t + 2 : t + 1, t + 1);
        return true;
    };

    // The others' shares.
    auto take = [&](const Tile& c, u64 t) {
        if (!wait_all([&](int p) { return done(p); }, t + 1, 61u)) return false;
        if (gathers) {
            constexpr int kBatch = 4;
            const unsigned rows = (unsigned)(n - 1) * c.rows;
            auto rank_of = [&](unsigned i) { return (r + 1 + (int)(i / c.rows)) % n; };
            for (unsigned i0 = warp; i0 < rows; i0 += kWarps * kBatch) {
                uint4 v[kBatch];
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const unsigned i = i0 + u * kWarps;
                    if (i < rows && (i % c.rows) * R::kSize + R::first(lane) < size_of(rank_of(i), c))
                        v[u] = ld16_host(result_slot(rank_of(i), t) + (i % c.rows) * 512u + lane * 16u);
                }
#pragma unroll
                for (int u = 0; u < kBatch; ++u) {
                    const unsigned i = i0 + u * kWarps;
                    if (i >= rows) break;
                    const int q = rank_of(i);
                    const unsigned e = (i % c.rows) * R::kSize + R::first(lane), size = size_of(q, c);
                    if (e < size) R::store(out, whole_at(q, c), e, size, lead, v[u]);
                }
            }
        }
        return true;
    };

    // This CTA's rows, in tiles that grow from first_rows and shrink towards the end: nothing can be read before the first tile
    // is given, and nothing is left to write while the last one is taken.
    const u64 row_end = a.rows * (u64)(cta + 1) / gridDim.x;
    auto tile_at = [&](u64 row0, unsigned after) {
        const u64 left = row_end > row0 ? row_end - row0 : 0;
        u64 rows = left / 2 > a.first_rows ? left / 2 : a.first_rows;
        if (rows > 2ull * after) rows = 2ull * after;
        if (rows > kHostChunkRows) rows = kHostChunkRows;
        return Tile{row0, (unsigned)(rows < left ? rows : left)};
    };
    Tile last{0, 0}, now = tile_at(a.rows * (u64)cta / gridDim.x, (a.first_rows + 1) / 2);
    u64 t = before;
    if (now.rows != 0) {
        if (reduces)
            for (unsigned i = warp; i < (unsigned)(n - 1) * now.rows; i += kWarps) give_store(give_load(i, now, t));
        publish(t + 1, t);
    }
    for (; now.rows != 0; ++t) {
        const Tile next = tile_at(now.row0 + now.rows, now.rows);
        if (!reduce(now, next, t)) return;  // the communicator is poisoned
        if (last.rows != 0 && !take(last, t - 1)) return;
        last = now;
        now = next;
    }
    if (last.rows != 0 && !take(last, t - 1)) return;
    __syncthreads();
    if (threadIdx.x == 0) *own_tiles = t;
}

template <typename T, typename Op>
cudaError_t start(bool wide, HostExchangeArgs& args, int ctas, cudaStream_t stream) {
    void* params[] = {&args};
    const void* kernel = wide ? reinterpret_cast<const void*>(host_exchange_kernel<T, Op, true>) : reinterpret_cast<const void*>(host_exchange_kernel<T, Op, false>);
    return cudaLaunchCooperativeKernel(kernel, dim3(ctas, args.nranks, 1), dim3(kThreads, 1, 1), params, 0, stream);
}

template <typename T>
cudaError_t start_op(RedOp op, bool wide, HostExchangeArgs& args, int ctas, cudaStream_t stream) {
    switch (op) {
        case RedOp::Sum:
        case RedOp::Avg: return start<T, OpAdd>(wide, args, ctas, stream);
        case RedOp::Max: return start<T, OpMax>(wide, args, ctas, stream);
        case RedOp::Min: return start<T, OpMin>(wide, args, ctas, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace

std::size_t host_parts_bytes(int nranks) { return std::size_t(nranks) * nranks * host_ctas(nranks) * kHostSlots * kHostChunkBytes; }
std::size_t host_results_bytes(int nranks) { return std::size_t(nranks) * host_ctas(nranks) * kHostSlots * kHostChunkBytes; }
std::size_t host_given_words(int nranks) { return std::size_t(nranks) * nranks * host_ctas(nranks); }
std::size_t host_done_words(int nranks) { return std::size_t(nranks) * host_ctas(nranks); }
std::size_t host_tiles_words(int nranks) { return std::size_t(nranks) * host_ctas(nranks); }

cudaError_t launch_host_exchange(DType dtype, RedOp op, bool wide, HostExchangeArgs args, cudaStream_t stream, int* used) {
    if (args.nranks < 2 || args.nranks > kMaxRanks) return cudaErrorInvalidValue;
    const u64 bytes = (args.count + args.lead) * dtype_size(dtype);
    args.rows = ring::div_up(bytes, ring::kGrainBytes * (args.collective == static_cast<int>(Collective::AllReduce) ? static_cast<u64>(args.nranks) : 1));
    args.first_rows = 128;  // 4 ranks, 4 MiB: 32 rows 751 us, 64 721, 128 704, 256 703; 8 ranks 1509, 1485, 1472, 1509
    args.ctas = host_ctas(args.nranks);
    const int ctas = static_cast<int>(std::min<u64>(host_ctas(args.nranks), std::max<u64>(1, args.rows / kWarps)));
    *used = ctas;
    switch (dtype) {
        case DType::Float: return start_op<float>(op, wide, args, ctas, stream);
        case DType::Float16: return start_op<__half>(op, wide, args, ctas, stream);
        case DType::BFloat16: return start_op<__nv_bfloat16>(op, wide, args, ctas, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace b200ccl::kernels
