// grid.cuh — the neighbour grid: cell keys, look-back scan, stable sort.
#pragma once

#include "common.cuh"

namespace fcu {

struct GridGeom {
    float min[3];
    float cell;
    uint32_t dims[3];
};

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;  // 4096 u32 per tile

constexpr int kRadixBits = 8;
constexpr uint32_t kRadix = 1u << kRadixBits;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;
constexpr uint32_t kSortTile = kSortThreads * kSortItems;  // 4096 keys per tile
constexpr int kMaxPasses = 4;                               // 32-bit keys
constexpr uint32_t kKeyBlocks = 148 * 8;                    // grid cap of the key kernels
#ifndef FCU_KEY_ITEMS
#define FCU_KEY_ITEMS 4
#endif
constexpr int kKeyItems = FCU_KEY_ITEMS;                    // positions per thread and round (cell keys; 498 us a 16.7M build at 4, 509 at 2, 516 at 8)

inline uint32_t div_up(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

// Digit passes for keys below `cells`.
inline int radix_passes(uint32_t cells) {
    uint32_t maxkey = cells > 0 ? cells - 1 : 0;
    int bits = 0;
    while (maxkey) {
        bits++;
        maxkey >>= 1;
    }
    int p = (bits + kRadixBits - 1) / kRadixBits;
    return p < 1 ? 1 : p;
}

// The first index of the sorted keys k[0 .. n) not below `key`, by a whole
// warp: 33 parts a round, so four rounds for a million keys.
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t *k, uint32_t n, uint32_t key) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, len = n;  // the answer is in lo .. lo + len
    while (len > 0) {
        const uint32_t step = len / 33 + 1;
        const uint64_t at = (uint64_t)lo + (uint64_t)step * (lane + 1) - 1;
        const bool below = at < lo + len && __ldcg(&k[at]) < key;
        const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, below));
        const uint32_t hi = lo + len;
        lo += c * step;
        len = min(step - 1, hi - lo);
    }
    return lo;
}

// Scratch of one grid build, carved from one device allocation.
// Words from the error word on that a build clears: the error word and, at
// kErrBarrier, the cooperative build's barrier counter.
constexpr uint32_t kErrWords = 32, kErrBarrier = 16;
struct GridWork {
    unsigned long long *scan_ctl;  // look-back words and digit counts, zeroed per build (or a cooperative build's piece counts)
    size_t scan_ctl_bytes;
    uint32_t *k1, *k2, *v1, *v2;   // ping-pong keys / values
    uint32_t *err;                 // device error word, and room for kErrWords from it
    int passes;
    uint32_t cells, n;
};

size_t grid_work_bytes(uint32_t n, uint32_t cells);
// Carves `ws` (at least grid_work_bytes) into a GridWork.
GridWork grid_work_carve(void *ws, uint32_t n, uint32_t cells, uint32_t *err);

// Reads a build's error word on `stream` (waiting for it): FLUID_OK, or
// FLUID_ERR_TIMEOUT with a reason when a bounded wait gave up (a look-back's,
// or the one-launch build's barrier).
int32_t read_build_status(const uint32_t *err, cudaStream_t stream, const char *who);
// Enqueues one block of a radix digit pass on the scratch of `w` (carved for
// at least two tiles of keys) that claims tile 1 while tile 0 never
// publishes: its bounded look-back waits give up and set w.err.
cudaError_t enqueue_stalled_radix_pass(const GridWork &w, cudaStream_t stream);

// The build in one cooperative launch (grid_coop.cu), for as many positions
// as one block per SM holds at once (1.2M positions) on the SMs that the
// stream may use.
constexpr uint32_t kCoopBlocks = 148;
bool coop_build_fits(const GridWork &w, cudaStream_t stream);
// cudaErrorCooperativeLaunchTooLarge, with nothing enqueued and no error left
// behind, where the driver would not hold every block at once after all.
cudaError_t coop_build_enqueue(cudaStream_t stream, const float4 *pos, const GridGeom &g, uint32_t *keys,
                               uint32_t *starts, uint32_t *perm, const GridWork &w);
// Enqueues the starts (starts[cells] = n) of the n sorted keys.
cudaError_t starts_enqueue(cudaStream_t stream, const uint32_t *sorted, uint32_t n, uint32_t cells, uint32_t *starts);
// Enqueues the same build with a barrier that expects an arrival more than
// come: every wait gives up and sets w.err.
cudaError_t enqueue_stalled_coop_build(cudaStream_t stream, const float4 *pos, const GridGeom &g, uint32_t *starts,
                                       uint32_t *perm, const GridWork &w);

// Enqueues keys -> stable radix sort -> starts on `stream`. `keys` receives
// each input's cell key, `starts` the exclusive scan of the cell counts with
// starts[cells] = n, `perm` the stable permutation. Clears the error word
// first.
cudaError_t grid_build_enqueue(cudaStream_t stream, const float4 *pos, uint32_t n, const GridGeom &g, uint32_t *keys,
                               uint32_t *starts, uint32_t *perm, GridWork &w);

// ---- the simulations' grid, by counting ----------------------------------------
// Keys are cell * kSimSlabs + x slab, so a cell's slots are in slab order.
constexpr int kCountThreads = 256;
constexpr int kCountItems = 4;  // positions per thread of the key kernel

// A batch of boxes sharing one grid: slot i belongs to box box_of[i], whose
// keys are cell_base[b] .. cell_base[b] + its cells * kSimSlabs - 1 (the
// boxes' key ranges laid end to end, in box order).
struct BoxKeys {
    const uint16_t *box_of;     // [n]
    const DevParams *box;       // [nboxes]
    const uint32_t *cell_base;  // [nboxes]
};

// Buffers of a counting build of `cells` keys: `count` and `ctl` are zero
// between builds (each build leaves them so), `order` holds indices below n.
struct CountGrid {
    uint32_t *keys, *count, *rank, *order, *starts, *perm;
    unsigned long long *ctl;  // the scan's look-back words
    uint32_t ctl_words;
    uint32_t *err;
    uint32_t n, cells;
};
// One allocation for count, rank, order and ctl; zero it once.
size_t count_grid_bytes(uint32_t n, uint32_t cells);
CountGrid count_grid_carve(void *ws, uint32_t n, uint32_t cells, uint32_t *keys, uint32_t *starts, uint32_t *perm,
                           uint32_t *err);

// What the key kernel does for the substep beside the keys: with `solve`,
// clears every box's residual accumulators, and with `ring` moves the
// substep's nboxes Step blocks (ring entry `cursor`) into cur[0 .. nboxes-1].
struct StepRing {
    const DevStep *ring = nullptr;
    DevStep *cur = nullptr;
    DevSolve *solve = nullptr;
    uint32_t size = 1, nboxes = 1;
};

// The particle records k_order moves into cell order with the permutation.
struct GridGather {
    const float4 *pos, *vel, *pvel;
    const float *pp, *temp;
    const uint32_t *id;
    float4 *wpos, *wvel, *wpvel;
    float *wpp, *wtemp;
    uint32_t *wid;
};

// Keys, starts (starts[cells] = n) and every index at a slot of its key's
// run; with `boxes` the keys are the batch's (`g` unused). n > 0.
cudaError_t count_grid_enqueue(cudaStream_t stream, const float4 *pos, const GridGeom &g, const BoxKeys *boxes,
                               const CountGrid &w, const StepRing &r);
// Enqueues one block of the scan that claims tile 1 while tile 0 never
// publishes: its bounded look-back gives up and sets w.err. The starts are
// invalid afterwards; counts and look-back words are left zero, as a build
// leaves them.
cudaError_t enqueue_stalled_scan(const CountGrid &w, cudaStream_t stream);
// Then the stable permutation and, with `gather`, the records in its order.
cudaError_t count_grid_order(cudaStream_t stream, const CountGrid &w, const GridGather *gather);

}  // namespace fcu
