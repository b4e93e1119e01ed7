// Rows: what a warp moves of a slice at a time, 32 vectors of 16 bytes, from and to a caller's buffer.
//
// 16-byte path (kWide): a lane's vector is 16 bytes of the buffer. Positions count from a 16-byte boundary, `lead` elements
// before the buffer (0 where it is aligned); those elements are never accessed. Otherwise a lane's vector is kElems elements that
// lie 32 apart, so that the warp's accesses are contiguous all the same at any alignment.
#pragma once

#include "kernels/sm100/vec.cuh"

namespace b200ccl::dev {

template <typename T, bool kWide>
struct Row {
    static constexpr int kElems = 16 / sizeof(T);
    static constexpr unsigned kSize = 32u * kElems;  // elements of a row
    static constexpr unsigned kStride = kWide ? 1u : 32u;

    // First element of a lane's vector, within the row; a lane without one has nothing in the row.
    static __device__ __forceinline__ unsigned first(unsigned lane) { return kWide ? lane * kElems : lane; }

    // Elements i0, i0 + kStride, ... of the slice of n elements that begins at `at`.
    static __device__ __forceinline__ uint4 load(const T* base, unsigned long long at, unsigned i0, unsigned n, unsigned lead) {
        if (kWide && i0 + kElems <= n && at + i0 >= lead) return ld16_stream(reinterpret_cast<const uint4*>(base + at + i0));
        T t[kElems];
#pragma unroll
        for (int e = 0; e < kElems; ++e) {
            const unsigned i = i0 + e * kStride;
            t[e] = Elem<T>::from_f(0.0f);
            if (i < n && (!kWide || at + i >= lead)) t[e] = Narrow<T>::load(base, at + i);
        }
        return *reinterpret_cast<const uint4*>(t);
    }
    static __device__ __forceinline__ void store(T* base, unsigned long long at, unsigned i0, unsigned n, unsigned lead, const uint4& v) {
        if (kWide && i0 + kElems <= n && at + i0 >= lead) {
            st16(reinterpret_cast<uint4*>(base + at + i0), v);
            return;
        }
        T t[kElems];
        *reinterpret_cast<uint4*>(t) = v;
#pragma unroll
        for (int e = 0; e < kElems; ++e) {
            const unsigned i = i0 + e * kStride;
            if (i < n && (!kWide || at + i >= lead)) base[at + i] = t[e];
        }
    }
};

}  // namespace b200ccl::dev
