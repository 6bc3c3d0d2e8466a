// wide.cuh — a particle shared by L adjacent lanes, its sums kept in order.
//
// The lanes form L pairs' terms at once and leave them in shared memory,
// term-major; lane a then adds term a of the L pairs in list order, so the
// additions of a chunk are chains that run side by side, one per lane. Empty
// places hold +0, which changes no sum (a sum that starts at +0 never becomes
// -0), so every sum is the one-thread loop's, bit for bit.
#pragma once

#include <stdint.h>

namespace fcu {

constexpr int kWideThreads = 128;
constexpr int kWideWarps = kWideThreads / 32;
// A term's row of 32 lanes, padded by 16 bytes so that the lanes of a group
// read their rows' 16-byte pieces from different banks.
template <class T>
constexpr int kRowOf = 32 + 16 / (int)sizeof(T);

// Lane `lane` of the group holding particle i. Every lane of a warp stays to
// the end; those past n work on the last particle with nothing to walk.
struct WideLane {
    uint32_t i, lane, group;  // group: the particle's place in its warp
    bool live;
};
template <int L>
__device__ __forceinline__ WideLane wide_lane(uint32_t n) {
    const uint32_t t = blockIdx.x * kWideThreads + threadIdx.x;
    const uint32_t i = t / L;
    return WideLane{i < n ? i : n - 1, t % L, (threadIdx.x & 31u) / L, i < n};
}

// acc plus the L values of a row's group, in order.
template <int L>
__device__ __forceinline__ float fold_row(float acc, const float *row) {
#pragma unroll
    for (int e = 0; e < L; e += 4) {
        const float4 q = *reinterpret_cast<const float4 *>(row + e);
        acc += q.x;
        acc += q.y;
        acc += q.z;
        acc += q.w;
    }
    return acc;
}
template <int L>
__device__ __forceinline__ double fold_row(double acc, const double *row) {
#pragma unroll
    for (int e = 0; e < L; e += 2) {
        const double2 q = *reinterpret_cast<const double2 *>(row + e);
        acc += q.x;
        acc += q.y;
    }
    return acc;
}

// The sums of R terms over a group's pairs: lane a keeps those of terms a,
// a + L, ...
template <class T, int L, int R>
struct WideSums {
    static constexpr int kPer = (R + L - 1) / L;
    T acc[kPer];
    __device__ __forceinline__ WideSums() {
#pragma unroll
        for (int q = 0; q < kPer; ++q) acc[q] = T(0);
    }
    // Adds one chunk: `rows` holds the warp's terms, written before a
    // __syncwarp by every lane.
    __device__ __forceinline__ void add(const T (*rows)[kRowOf<T>], const WideLane &w) {
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const int a = (int)w.lane + q * L;
            if (a < R) acc[q] = fold_row<L>(acc[q], rows[a] + w.group * L);
        }
    }
    // Term A's sum, on every lane of the group.
    template <int A>
    __device__ __forceinline__ T get() const {
        return __shfl_sync(0xffffffffu, acc[A / L], A % L, L);
    }
};

// The candidates of nine stencil rows, L at a time in stencil order: a
// group's lanes stand at consecutive candidates of its rows (beg, len in
// shared memory) laid end to end.
struct WideRows {
    const uint32_t *beg, *len;
    uint32_t row, off;
    __device__ __forceinline__ WideRows(const uint32_t *b, const uint32_t *l, uint32_t lane)
        : beg(b), len(l), row(0), off(lane) {
        settle();
    }
    __device__ __forceinline__ void settle() {
        while (row < 9u && off >= len[row]) {
            off -= len[row];
            ++row;
        }
    }
    __device__ __forceinline__ bool any() const { return row < 9u; }
    __device__ __forceinline__ uint32_t at() const { return beg[row] + off; }
    template <int L>
    __device__ __forceinline__ void next() {
        off += L;
        settle();
    }
};
constexpr uint32_t kWideStage = 64;  // hits staged before they are processed
template <int L>
constexpr int kWideLoads = L >= 32 ? 2 : 4;  // candidates a lane loads before testing any
template <int L>
constexpr int kWideCap = (int)kWideStage + L * kWideLoads<L>;  // staged hits at most
// The lanes of this lane's group, in a warp-wide mask.
template <int L>
__device__ __forceinline__ uint32_t group_mask(const WideLane &w) {
    return L == 32 ? 0xffffffffu : ((1u << (L & 31)) - 1u) << (w.group * L);
}

}  // namespace fcu
