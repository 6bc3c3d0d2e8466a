// grid.cu — neighbour grid build for sm_100a.
//
// Reference: count / scatter in crates/fluid-core/src/sim_grid.wgsl:36-72 and
// sim_density.wgsl:36-55; the scan in sim_scan.wgsl:97-120 (exclusive, with
// the total at starts[cells]). The reference's scatter ranks particles inside
// a cell by atomic arrival; this build is stable (ascending input index inside
// a cell), the order a sequential counting sort produces.
//
//   k_cell_keys      key = cell_of(pos), and every radix pass's digit
//                    counts over all keys
//   k_radix_pass     one stable 8-bit digit pass: warp ranking in input
//                    order (digit peers from eight ballots), the tile staged
//                    in shared memory in digit order, its digit offsets by
//                    decoupled look-back over the earlier tiles, written out
//                    coalesced; every spin is bounded
//   k_starts         starts from the sorted keys, tile of cells by tile
//
// Up to 1.2M positions the build is grid_coop.cu's single launch instead.
// A simulation's own grid (keys of cell and x slab, few particles a key) is
// built by counting instead: k_count_keys, k_scan_lookback (a single-pass
// exclusive scan, decoupled look-back with bounded spins), k_place, k_order.
#include <algorithm>
#include <string>

#include "grid.cuh"

namespace fcu {

namespace {

constexpr unsigned long long kFlagAgg = 1ull << 32;
constexpr unsigned long long kFlagPrefix = 2ull << 32;

__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The lanes of `act` whose 8-bit digit equals this lane's: what
// __match_any_sync(act, d) returns, from one ballot per digit bit (a build of
// 16.7M positions 498 us, by the general match 644). Every lane of the warp
// calls it.
__device__ __forceinline__ uint32_t digit_peers(uint32_t act, uint32_t d) {
    uint32_t m = act;
#pragma unroll
    for (int b = 0; b < kRadixBits; ++b) {
        const uint32_t bit = (d >> b) & 1u;
        const uint32_t bal = __ballot_sync(0xffffffffu, bit);
        m &= bit ? bal : ~bal;
    }
    return m;
}

// Every pass's digit counts over all keys: a block's shared histograms,
// then one global add per nonzero bin. One shared add a key and digit: the
// unit merges the adds of equal digits in a warp, so that finding runs of
// them first only cost (the kernel 109 -> 68 us at 16.7M positions in
// any order).
__device__ __forceinline__ void count_digits(uint32_t (*h)[kRadix], int passes, uint32_t key) {
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(key >> (p * kRadixBits)) & (kRadix - 1)], 1u);
}
__device__ __forceinline__ void flush_digits(uint32_t (*h)[kRadix], int passes, uint32_t *digit_counts) {
    __syncthreads();
    for (int p = 0; p < passes; ++p) {
        const uint32_t c = h[p][threadIdx.x];
        if (c) atomicAdd(&digit_counts[p * kRadix + threadIdx.x], c);
    }
}

// Cell key of every position, and every radix pass's digit counts. A
// grid-stride loop over a capped grid, so the digit counts leave each block
// once.
__global__ void __launch_bounds__(kSortThreads) k_cell_keys(const float4 *__restrict__ pos, uint32_t n,
                                                            GridGeom g, uint32_t *__restrict__ keys,
                                                            int passes, uint32_t *digit_counts) {
    __shared__ uint32_t h[kMaxPasses][kRadix];
    for (int p = 0; p < kMaxPasses; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    // kKeyItems positions per thread and round, all loaded before any is used
    const uint64_t stride = (uint64_t)gridDim.x * kSortThreads * kKeyItems;
    for (uint64_t at = (uint64_t)blockIdx.x * kSortThreads * kKeyItems; at < n; at += stride) {
        float4 p[kKeyItems];
#pragma unroll
        for (int u = 0; u < kKeyItems; ++u) {
            const uint64_t i = at + (uint64_t)u * kSortThreads + threadIdx.x;
            p[u] = i < n ? __ldg(&pos[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < kKeyItems; ++u) {
            const uint64_t i = at + (uint64_t)u * kSortThreads + threadIdx.x;
            if (i < n) {
                const uint32_t cx = axis_cell(p[u].x, g.min[0], g.cell, g.dims[0]);
                const uint32_t cy = axis_cell(p[u].y, g.min[1], g.cell, g.dims[1]);
                const uint32_t cz = axis_cell(p[u].z, g.min[2], g.cell, g.dims[2]);
                const uint32_t key = (cz * g.dims[1] + cy) * g.dims[0] + cx;
                keys[i] = key;
                count_digits(h, passes, key);
            }
        }
    }
    flush_digits(h, passes, digit_counts);
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Exclusive sums of in[0..n) into out[0..n), single pass. Tiles are claimed in launch order through ctl[0];
// ctl[1 + t] is tile t's status word: flag in the high half (1 aggregate,
// 2 inclusive prefix), value in the low half. With write_total, out[n]
// receives the grand total. With zero_in, the input is cleared after it is
// read.
__global__ void __launch_bounds__(kScanThreads) k_scan_lookback(uint32_t *in, uint32_t *out,
                                                                uint32_t n,
                                                                unsigned long long *ctl,
                                                                uint32_t *err, int write_total,
                                                                int zero_in) {
    __shared__ uint32_t s_tile;
    __shared__ uint32_t s_warp[kScanThreads / 32];
    __shared__ uint32_t s_excl;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd((unsigned int *)ctl, 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    unsigned long long *status = ctl + 1;
    const uint64_t base = (uint64_t)tile * kScanTile + (uint64_t)threadIdx.x * kScanItems;

    uint32_t v[kScanItems];
    const bool vec = base + kScanItems <= n && ((uintptr_t)(in + base) & 15u) == 0 &&
                     ((uintptr_t)(out + base) & 15u) == 0;
    if (vec) {
        const uint4 *src = reinterpret_cast<const uint4 *>(in + base);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q) {
            const uint4 x = src[q];
            v[4 * q + 0] = x.x;
            v[4 * q + 1] = x.y;
            v[4 * q + 2] = x.z;
            v[4 * q + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = (base + k < n) ? in[base + k] : 0u;
    }
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) sum += v[k];

    // block-wide scan of the thread sums
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    uint32_t x_before = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) x_before = 0u;
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kScanThreads / 32 ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < kScanThreads / 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += y;
        }
        if (lane < kScanThreads / 32) s_warp[lane] = w;
    }
    __syncthreads();
    const uint32_t block_total = s_warp[kScanThreads / 32 - 1];
    const uint32_t thread_excl = (warp > 0 ? s_warp[warp - 1] : 0u) + x_before;

    // decoupled look-back, warp 0
    if (warp == 0) {
        uint32_t exclusive = 0;
        if (tile == 0) {
            if (lane == 0) st_relaxed(&status[0], kFlagPrefix | block_total);
        } else {
            if (lane == 0) st_relaxed(&status[tile], kFlagAgg | block_total);
            int64_t pred = (int64_t)tile - 1;
            while (true) {
                const int64_t idx = pred - (int64_t)lane;
                unsigned long long st = idx >= 0 ? ld_relaxed(&status[idx]) : kFlagPrefix;
                uint32_t spins = 0;
                while (true) {
                    const bool invalid = (st >> 32) == 0;
                    if (!__any_sync(0xffffffffu, invalid)) break;
                    if (++spins > kSpinLimit) {
                        if (lane == 0) atomicOr(err, ERRF_SCAN_TIMEOUT);
                        if (invalid) st = kFlagPrefix;  // give up: count it as zero
                        break;
                    }
                    if (invalid) st = ld_relaxed(&status[idx]);
                }
                const uint32_t pmask = __ballot_sync(0xffffffffu, (st >> 32) == 2ull);
                const uint32_t val = (uint32_t)st;
                if (pmask) {
                    const int j = __ffs(pmask) - 1;
                    exclusive += warp_sum((int)lane <= j ? val : 0u);
                    break;
                }
                exclusive += warp_sum(val);
                pred -= 32;
            }
            if (lane == 0)
                st_relaxed(&status[tile], kFlagPrefix | (unsigned long long)(exclusive + block_total));
        }
        if (lane == 0) s_excl = exclusive;
    }
    __syncthreads();
    uint32_t run = s_excl + thread_excl;
    if (vec) {
        uint32_t o[kScanItems];
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            o[k] = run;
            run += v[k];
        }
        uint4 *dst = reinterpret_cast<uint4 *>(out + base);
#pragma unroll
        for (int q = 0; q < kScanItems / 4; ++q)
            dst[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
        if (zero_in) {
            uint4 *z = reinterpret_cast<uint4 *>(in + base);
#pragma unroll
            for (int q = 0; q < kScanItems / 4; ++q) z[q] = make_uint4(0, 0, 0, 0);
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (base + k < n) {
                out[base + k] = run;
                if (zero_in) in[base + k] = 0u;
            }
            run += v[k];
        }
    }
    if (write_total && threadIdx.x == 0 && (uint64_t)(tile + 1) * kScanTile >= n)
        out[n] = s_excl + block_total;
}

// One stable digit pass. Tiles are claimed in launch order through
// *tile_ctr. Warp w of tile t owns the contiguous run t*TILE + w*32*ITEMS ..
// +32*ITEMS; in round r lane l holds element run + r*32 + l, so (warp,
// round, lane) is input order and ranks taken in that order keep equal
// digits in input order. The tile's count of each digit d is published in
// tile_status[t][d] (flag in the high half: 1 this tile's count, 2 the
// inclusive count over tiles 0..t), and the thread of digit d looks back
// over the tiles before it for their counts of d (decoupled look-back, one
// chain per digit, every spin bounded). A digit's output run starts at the
// number of smaller digits over all keys (digit_counts) plus its count in
// earlier tiles. The tile is laid out in shared memory in (digit, input)
// order and written out by consecutive threads to consecutive addresses.
// `vals_in` null means the identity (the first pass).
static_assert(kRadix == kSortThreads, "one thread per digit");
// Blocks per SM the pass kernel is compiled for: 498 us a build of 16.7M
// positions at 4 (64 registers), 538 at 3, 577 at 5 (spills). Of a form of the
// build that took 522: tiles of 8,192 keys by 512 threads 539, of 16,384 by
// 1,024 604, of 3,072 by 256 558.
#ifndef FCU_SORT_MINB
#define FCU_SORT_MINB 4
#endif
// FCU_VAL_PREFETCH > 0: a digit pass asks L1 for the values of every
// FCU_VAL_PREFETCH-th round of its tile while it ranks the keys: 539 us a
// build of 16.7M positions without, 498 at 1.
#ifndef FCU_VAL_PREFETCH
#define FCU_VAL_PREFETCH 1
#endif
// Earlier tiles' status words a digit's look-back loads at once: 503 us a
// build of 16.7M positions at 2, 498 at 4, 512 at 8 (spills).
#ifndef FCU_LOOK_WINDOW
#define FCU_LOOK_WINDOW 4
#endif
constexpr int kLookWindow = FCU_LOOK_WINDOW;

__global__ void __launch_bounds__(kSortThreads, FCU_SORT_MINB) k_radix_pass(
    const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in, uint32_t n, int shift,
    const uint32_t *__restrict__ digit_counts, unsigned long long *tile_status, uint32_t *tile_ctr,
    uint32_t *err, uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out) {
    __shared__ uint32_t s_hist[kSortWarps][kRadix];
    __shared__ uint32_t s_off[kRadix];    // output index of this tile's first element of digit d
    __shared__ uint32_t s_start[kRadix];  // staged index of the tile's first element of digit d
    __shared__ uint32_t s_wsum[kSortWarps];
    __shared__ uint32_t s_gsum[kSortWarps];
    __shared__ uint32_t s_key[kSortTile];
    __shared__ uint32_t s_val[kSortTile];
    __shared__ uint32_t s_tile;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr, 1u);
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s_hist[w][threadIdx.x] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;

    // Indices fit 32 bits: the last tile ends at ceil(n / kSortTile) *
    // kSortTile <= 2^32 for any 32-bit n. A full tile (every tile but the
    // last) takes the loads and ballots without per-element bounds.
    const uint32_t wbase = tile * kSortTile + warp * (32 * kSortItems);
    const bool full = (uint64_t)(tile + 1) * kSortTile <= n;
    const uint32_t lt = lanemask_lt();
    uint32_t key[kSortItems], rank[kSortItems];
    if (full) {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) key[r] = __ldg(&keys_in[wbase + r * 32 + lane]);
    } else {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t i = wbase + r * 32 + lane;
            key[r] = i < n ? __ldg(&keys_in[i]) : 0u;
        }
    }
#if FCU_VAL_PREFETCH
    // the values are read only after the ranking and the look-back: ask L1
    // for them now (no registers held) so that read finds them there
    if (vals_in) {
#pragma unroll
        for (int r = 0; r < kSortItems; r += FCU_VAL_PREFETCH) {
            const uint32_t i = wbase + r * 32 + lane;
            if (full || i < n) asm volatile("prefetch.global.L1 [%0];" ::"l"(vals_in + i));
        }
    }
#endif
    // every round's digit peers first (ballots and registers only), then the
    // rounds in order: the leader of each group of peers adds the group to
    // the warp's count of its digit and hands the old count to the group
    if (full) {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const uint32_t d = (key[r] >> shift) & (kRadix - 1);
            rank[r] = digit_peers(0xffffffffu, d);
        }
    } else {
#pragma unroll
        for (int r = 0; r < kSortItems; ++r) {
            const bool live = wbase + r * 32 + lane < n;
            const uint32_t act = __ballot_sync(0xffffffffu, live);
            const uint32_t d = (key[r] >> shift) & (kRadix - 1);
            const uint32_t pe = digit_peers(act, d);
            rank[r] = live ? pe : 0u;  // a live lane is its own peer, so nonzero
        }
    }
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t peers = rank[r];
        const uint32_t d = (key[r] >> shift) & (kRadix - 1);
        const uint32_t leader = peers ? (uint32_t)(__ffs(peers) - 1) : lane;
        uint32_t before = 0;
        if (peers && lane == leader) before = atomicAdd(&s_hist[warp][d], (uint32_t)__popc(peers));
        before = __shfl_sync(0xffffffffu, before, leader);
        rank[r] = before + __popc(peers & lt);
        __syncwarp();  // this round's adds land before the next round's
    }
    __syncthreads();
    // thread = digit d: the warps' exclusive counts of it, and its tile count
    const uint32_t dig = threadIdx.x;
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t t = s_hist[w][dig];
        s_hist[w][dig] = total;
        total += t;
    }
    unsigned long long *mine = tile_status + (uint64_t)tile * kRadix;
    st_relaxed(&mine[dig], (tile == 0 ? kFlagPrefix : kFlagAgg) | total);

    // exclusive scans over the digits: of the tile counts (staged starts)
    // and of the global counts (where each digit's output begins)
    const uint32_t gc = __ldg(&digit_counts[dig]);
    uint32_t x = total, y = gc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t xu = __shfl_up_sync(0xffffffffu, x, o);
        const uint32_t yu = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= (uint32_t)o) {
            x += xu;
            y += yu;
        }
    }
    if (lane == 31) {
        s_wsum[warp] = x;
        s_gsum[warp] = y;
    }

    __syncthreads();
    uint32_t wx = 0, wy = 0;
    for (uint32_t w = 0; w < warp; ++w) {
        wx += s_wsum[w];
        wy += s_gsum[w];
    }
    s_start[dig] = wx + x - total;
    __syncthreads();
    // staged while the earlier tiles publish their counts (behind the
    // look-back instead: 149 us a pass at 16.7M positions, 125 so)
#pragma unroll
    for (int r = 0; r < kSortItems; ++r) {
        const uint32_t i = wbase + r * 32 + lane;
        if (full || i < n) {
            const uint32_t d = (key[r] >> shift) & (kRadix - 1);
            const uint32_t at = s_start[d] + s_hist[warp][d] + rank[r];
            s_key[at] = key[r];
            s_val[at] = vals_in ? __ldg(&vals_in[i]) : i;
        }
    }

    // look-back over the earlier tiles' counts of this digit: the status
    // words of kLookWindow earlier tiles are loaded at once, then taken in
    // order (an entry read while unpublished is re-read until it is), adding
    // counts until the first inclusive one. A word read early as a tile's own
    // count is still that count, so the sum is the same as one tile at a
    // time; only the chain of L2 round trips is shorter (a single wave of
    // tiles, as at 1M keys, otherwise walks back one tile per round trip).
    uint32_t excl = 0;
    if (tile > 0) {
        int64_t pred = (int64_t)tile - 1;
        bool done = false;
        while (!done) {
            unsigned long long v[kLookWindow];
#pragma unroll
            for (int u = 0; u < kLookWindow; ++u)
                v[u] = pred - u >= 0 ? ld_relaxed(&tile_status[(uint64_t)(pred - u) * kRadix + dig]) : kFlagPrefix;
#pragma unroll
            for (int u = 0; u < kLookWindow; ++u) {
                if (done) continue;
                unsigned long long st = v[u];
                uint32_t spins = 0;
                while ((st >> 32) == 0) {
                    if (++spins > kSpinLimit) {
                        atomicOr(err, ERRF_SCAN_TIMEOUT);
                        st = kFlagPrefix;  // give up: count it as zero and stop
                        break;
                    }
                    st = ld_relaxed(&tile_status[(uint64_t)(pred - u) * kRadix + dig]);
                }
                excl += (uint32_t)st;
                if ((st >> 32) == 2ull) done = true;
            }
            pred -= kLookWindow;
        }
        st_relaxed(&mine[dig], kFlagPrefix | (unsigned long long)(excl + total));
    }
    s_off[dig] = wy + y - gc + excl;
    __syncthreads();
    const uint32_t tbase = tile * kSortTile;
    const uint32_t count = full ? kSortTile : n - tbase;
    for (uint32_t j = threadIdx.x; j < count; j += kSortThreads) {
        const uint32_t k = s_key[j];
        const uint32_t d = (k >> shift) & (kRadix - 1);
        const uint32_t dst = s_off[d] + (j - s_start[d]);
        // Always below n when the counts are right; the test keeps a
        // look-back that gave up (garbage offsets) from writing out of bounds.
        if (dst < n) {
            vals_out[dst] = s_val[j];
            keys_out[dst] = k;
        }
    }
}

// The starts from the sorted keys. A block takes kStartTile cells, finds
// their range of keys by two searches, marks the end of every run of equal
// keys in shared memory and carries the marks over the empty cells by a
// block-wide max scan, so nothing waits on another block. Where the range is
// many keys for its cells (kStartStream), each cell's start is searched
// instead, four cells of a thread side by side: all keys in one cell then
// cost no more than the searches. The look-back max scan this replaces, over
// run ends that the last digit pass scattered into cleared starts, took 65 us
// at 2^24 cells, with its memset 80; this takes 45.
constexpr int kStartThreads = 256, kStartSearch = 4, kStartMinBlocks = 6;
constexpr uint32_t kStartStream = 65536;

template <int kStartItems>
__global__ void __launch_bounds__(kStartThreads, kStartMinBlocks)
    k_starts(const uint32_t *__restrict__ sorted, uint32_t n, uint32_t cells, uint32_t *__restrict__ starts) {
    constexpr uint32_t kStartTile = kStartThreads * kStartItems;
    __shared__ uint32_t s_end[kStartTile + kStartThreads];
    auto start_word = [](uint32_t x) { return x + x / kStartItems; };  // no bank conflicts
    __shared__ uint32_t s_bound[2], s_warp[kStartThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t c0 = blockIdx.x * kStartTile, count = min(kStartTile, cells - c0);
    if (warp < 2) {
        // (a bound past the last cell is above every key)
        const uint32_t at = warp_lower_bound(sorted, n, warp ? c0 + count : c0);
        if (lane == 0) s_bound[warp] = at;
    }
    for (uint32_t x = tid; x < kStartTile + kStartThreads; x += kStartThreads) s_end[x] = 0u;
    __syncthreads();
    const uint32_t lo = s_bound[0], hi = max(s_bound[1], lo);
    if (blockIdx.x == gridDim.x - 1 && tid == 0) starts[cells] = n;
    if (hi - lo > kStartStream) {
        for (uint32_t x0 = tid; x0 < count; x0 += kStartSearch * kStartThreads) {
            uint32_t at[kStartSearch];
#pragma unroll
            for (int u = 0; u < kStartSearch; ++u) at[u] = lo;
            // the answer is in at .. at + len; the same len for all
            for (uint32_t len = hi - lo; len > 0;) {
                const uint32_t half = len >> 1;
#pragma unroll
                for (int u = 0; u < kStartSearch; ++u) {
                    const bool below = __ldg(&sorted[at[u] + half]) < c0 + x0 + u * kStartThreads;
                    at[u] = below ? at[u] + len - half : at[u];
                }
                len = half;
            }
#pragma unroll
            for (int u = 0; u < kStartSearch; ++u)
                if (x0 + u * kStartThreads < count) starts[c0 + x0 + u * kStartThreads] = at[u];
        }
        return;
    }
#pragma unroll 4
    for (uint32_t j = lo + tid; j < hi; j += kStartThreads) {
        const uint32_t k = __ldg(&sorted[j]);
        const uint32_t kn = j + 1 < hi ? __ldg(&sorted[j + 1]) : ~k;
        const uint32_t x = k - c0;
        if (kn != k && x < count) s_end[start_word(x)] = j + 1;  // (x is below count unless a digit pass gave up)
    }
    __syncthreads();
    uint32_t v[kStartItems];
    uint32_t top = 0;
#pragma unroll
    for (int u = 0; u < kStartItems; ++u) {
        v[u] = s_end[start_word(tid * kStartItems + u)];
        top = max(top, v[u]);
    }
    uint32_t x = top;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x = max(x, y);
    }
    uint32_t run = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) run = 0u;
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    run = max(run, lo);
    for (uint32_t w = 0; w < warp; ++w) run = max(run, s_warp[w]);
#pragma unroll
    for (int u = 0; u < kStartItems; ++u) {
        s_end[start_word(tid * kStartItems + u)] = run;
        run = max(run, v[u]);
    }
    __syncthreads();
    for (uint32_t y = tid; y < count; y += kStartThreads) starts[c0 + y] = s_end[start_word(y)];
}

// ---- the counting build of the simulations ------------------------------------
// k_count_keys, an exclusive scan of the counts, k_place and k_order. A
// simulation's cells hold a few particles each (13 of them, 3 a slab, in
// water at rest), so instead of three digit passes over all keys its
// particles are counted per key, placed at their key's start in the order
// their atomics arrived, and each then finds its place inside its key's run
// by counting the run's smaller slots: the stable order, whatever the
// arrival. A particle's look through its run is a fraction of its look
// through its whole stencil in the density sweep after it, also where a
// clump makes runs long. Measured against the digit passes, keys to gathered
// records: 140 -> 70 us at 1,048,576 particles over 4.4M keys, 85 -> 35 at
// 152,559, 75 -> 29 at 72,072, 51 -> 29 at 1,620 (a substep 123 -> 104 us).
// What is left: the scan's pass over the keys and the records' 128 bytes a
// particle at the large end, four launches at the small one.

// Key of every position, and its arrival rank among the positions of its
// key: one add per run of equal keys in adjacent lanes (positions are nearly
// in cell order, so runs are long). The grid's first threads also move the
// substep's Step blocks from the ring into `cur` and clear the residual
// accumulators.
template <bool kBoxes>
__global__ void __launch_bounds__(kCountThreads) k_count_keys(const float4 *__restrict__ pos, GridGeom g,
                                                              BoxKeys bk, CountGrid w, StepRing r) {
    const uint32_t n = w.n;
    if (r.solve) {
        const uint32_t t = blockIdx.x * kCountThreads + threadIdx.x;
        for (uint32_t q = t; q < r.nboxes * 2u * kAccSlots; q += gridDim.x * kCountThreads)
            r.solve[q / (2u * kAccSlots)].acc_div[q % (2u * kAccSlots)] = 0ull;  // acc_div, then acc_den
        if (r.ring && blockIdx.x == 0) {
            const uint32_t c = r.solve->cursor;
            const DevStep *src = r.ring + (size_t)(c % r.size) * r.nboxes;
            for (uint32_t b = threadIdx.x; b < r.nboxes; b += kCountThreads) r.cur[b] = src[b];
            __syncthreads();  // every thread has read the cursor before it moves
            if (threadIdx.x == 0) r.solve->cursor = c + 1u;
        }
    }
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t at = blockIdx.x * (kCountThreads * kCountItems) + threadIdx.x;
    float4 p[kCountItems];
#pragma unroll
    for (int u = 0; u < kCountItems; ++u) {
        const uint32_t i = at + u * kCountThreads;
        p[u] = i < n ? __ldg(&pos[i]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kCountItems; ++u) {
        const uint32_t i = at + u * kCountThreads;
        const bool live = i < n;
        uint32_t key = 0xffffffffu;  // no key: keys stay below it
        if (live) {
            if (kBoxes) {
                const uint32_t b = __ldg(&bk.box_of[i]);
                const DevParams *P = &bk.box[b];
                const float cell = __ldg(&P->cell), mx = __ldg(&P->box_min[0]);
                const uint32_t dx = __ldg(&P->dims[0]), dy = __ldg(&P->dims[1]), dz = __ldg(&P->dims[2]);
                const uint32_t cx = axis_cell(p[u].x, mx, cell, dx);
                const uint32_t cy = axis_cell(p[u].y, __ldg(&P->box_min[1]), cell, dy);
                const uint32_t cz = axis_cell(p[u].z, __ldg(&P->box_min[2]), cell, dz);
                key = ((cz * dy + cy) * dx + cx) * kSimSlabs + axis_slab(p[u].x, mx, cell, cx, kSimSlabs) +
                      __ldg(&bk.cell_base[b]);
            } else {
                const uint32_t cx = axis_cell(p[u].x, g.min[0], g.cell, g.dims[0]);
                const uint32_t cy = axis_cell(p[u].y, g.min[1], g.cell, g.dims[1]);
                const uint32_t cz = axis_cell(p[u].z, g.min[2], g.cell, g.dims[2]);
                key = ((cz * g.dims[1] + cy) * g.dims[0] + cx) * kSimSlabs +
                      axis_slab(p[u].x, g.min[0], g.cell, cx, kSimSlabs);
            }
        }
        const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
        const bool head = lane == 0 || prev != key;
        const uint32_t heads = __ballot_sync(0xffffffffu, head);
        const uint32_t first = 31u - (uint32_t)__clz(heads & (0xffffffffu >> (31u - lane)));
        const uint32_t after = heads & ~(0xffffffffu >> (31u - lane));
        uint32_t base = 0;
        if (head && live) base = atomicAdd(&w.count[key], (after ? (uint32_t)__ffs(after) - 1u : 32u) - lane);
        base = __shfl_sync(0xffffffffu, base, first);
        if (live) {
            w.keys[i] = key;
            w.rank[i] = base + lane - first;
        }
    }
}

// Each index at its key's start plus its arrival rank.
__global__ void __launch_bounds__(kCountThreads) k_place(CountGrid w) {
    const uint32_t i = blockIdx.x * kCountThreads + threadIdx.x;
    if (i >= w.n) return;
    const uint32_t slot = __ldg(&w.starts[__ldg(&w.keys[i])]) + __ldg(&w.rank[i]);
    if (slot < w.n) w.order[slot] = i;  // always, unless the scan gave up
}

// The index placed at this thread's slot goes to its key's start plus the
// number of smaller indices in the key's run, and with kGather the
// particle's records with it. Also clears the scan's control words for the
// next build.
template <bool kGather>
__global__ void __launch_bounds__(kCountThreads) k_order(CountGrid w, GridGather a) {
    const uint32_t t = blockIdx.x * kCountThreads + threadIdx.x;
    for (uint32_t q = t; q < w.ctl_words; q += gridDim.x * kCountThreads) w.ctl[q] = 0ull;
    if (t >= w.n) return;
    const uint32_t i = __ldg(&w.order[t]);
    const uint32_t c = __ldg(&w.keys[i]);
    const uint32_t s = __ldg(&w.starts[c]);
    const uint32_t e = min(__ldg(&w.starts[c + 1]), w.n);
    float4 pos, vel, pvel;
    float pp, temp;
    uint32_t id;
    if (kGather) {
        pos = __ldg(&a.pos[i]);
        vel = __ldg(&a.vel[i]);
        pvel = __ldg(&a.pvel[i]);
        pp = __ldg(&a.pp[i]);
        temp = __ldg(&a.temp[i]);
        id = __ldg(&a.id[i]);
    }
    uint32_t dst = s;
    for (uint32_t k = s; k < e; k += 4) {
        uint32_t o[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) o[u] = k + u < e ? __ldg(&w.order[k + u]) : i;
#pragma unroll
        for (int u = 0; u < 4; ++u) dst += o[u] < i ? 1u : 0u;
    }
    if (dst >= w.n) return;  // only after a scan that gave up
    w.perm[dst] = i;
    if (kGather) {
        a.wpos[dst] = pos;
        a.wvel[dst] = vel;
        a.wpvel[dst] = pvel;
        a.wpp[dst] = pp;
        a.wtemp[dst] = temp;
        a.wid[dst] = id;
    }
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

size_t scan_region_bytes(uint32_t len) {
    return align256(8ull * (1ull + div_up(len, kScanTile)));
}

__global__ void k_fill_u32(uint32_t *p, uint32_t n, uint32_t v) {
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) p[i] = v;
}

// The zeroed part of the workspace: every pass's tile counter and tile status
// words, every pass's digit counts.
struct SortRegion {
    uint32_t *tile_ctr[kMaxPasses];
    unsigned long long *tile_status[kMaxPasses];
    uint32_t *digit_counts;
    size_t bytes;
};

SortRegion sort_region(void *base, uint32_t n, uint32_t cells, int passes) {
    SortRegion r{};
    const uint32_t tiles = div_up(n > 0 ? n : 1, kSortTile);
    const uintptr_t b = reinterpret_cast<uintptr_t>(base);
    size_t off = 0;
    off += scan_region_bytes(cells + 1);  // room for a cooperative build's piece counts
    for (int q = 0; q < passes; ++q) {
        r.tile_ctr[q] = reinterpret_cast<uint32_t *>(b + off);
        off += 256;
        r.tile_status[q] = reinterpret_cast<unsigned long long *>(b + off);
        off += align256(8ull * kRadix * tiles);
    }
    r.digit_counts = reinterpret_cast<uint32_t *>(b + off);
    off += align256(4ull * kRadix * kMaxPasses);
    r.bytes = off;
    return r;
}

}  // namespace

size_t grid_work_bytes(uint32_t n, uint32_t cells) {
    size_t b = sort_region(nullptr, n, cells, radix_passes(cells)).bytes;
    b += 4 * align256(4ull * (n > 0 ? n : 1));
    b += 256;  // err word when the caller gives none
    return b;
}

GridWork grid_work_carve(void *ws, uint32_t n, uint32_t cells, uint32_t *err) {
    GridWork w{};
    w.passes = radix_passes(cells);
    w.cells = cells;
    w.n = n;
    char *p = (char *)ws;
    w.scan_ctl = (unsigned long long *)p;
    w.scan_ctl_bytes = sort_region(ws, n, cells, w.passes).bytes;
    p += w.scan_ctl_bytes;
    const size_t nb = align256(4ull * (n > 0 ? n : 1));
    w.k1 = (uint32_t *)p;
    p += nb;
    w.k2 = (uint32_t *)p;
    p += nb;
    w.v1 = (uint32_t *)p;
    p += nb;
    w.v2 = (uint32_t *)p;
    p += nb;
    w.err = err ? err : (uint32_t *)p;
    return w;
}

size_t count_grid_bytes(uint32_t n, uint32_t cells) {
    return scan_region_bytes(cells) + align256(4ull * cells) + 2 * align256(4ull * n);
}

CountGrid count_grid_carve(void *ws, uint32_t n, uint32_t cells, uint32_t *keys, uint32_t *starts, uint32_t *perm,
                           uint32_t *err) {
    CountGrid w{};
    char *p = (char *)ws;
    w.ctl = (unsigned long long *)p;
    w.ctl_words = 1u + div_up(cells, kScanTile);
    p += scan_region_bytes(cells);
    w.count = (uint32_t *)p;
    p += align256(4ull * cells);
    w.rank = (uint32_t *)p;
    p += align256(4ull * n);
    w.order = (uint32_t *)p;
    w.keys = keys;
    w.starts = starts;
    w.perm = perm;
    w.err = err;
    w.n = n;
    w.cells = cells;
    return w;
}

cudaError_t count_grid_enqueue(cudaStream_t stream, const float4 *pos, const GridGeom &g, const BoxKeys *boxes,
                               const CountGrid &w, const StepRing &r) {
    const uint32_t blocks = div_up(w.n, kCountThreads * kCountItems);
    if (boxes) k_count_keys<true><<<blocks, kCountThreads, 0, stream>>>(pos, g, *boxes, w, r);
    else k_count_keys<false><<<blocks, kCountThreads, 0, stream>>>(pos, g, BoxKeys{}, w, r);
    k_scan_lookback<<<div_up(w.cells, kScanTile), kScanThreads, 0, stream>>>(w.count, w.starts, w.cells, w.ctl,
                                                                                   w.err, 1, 1);
    k_place<<<div_up(w.n, kCountThreads), kCountThreads, 0, stream>>>(w);
    return cudaGetLastError();
}

cudaError_t enqueue_stalled_scan(const CountGrid &w, cudaStream_t st) {
    // the tile counter starts at 1, so the one block claims tile 1 (of no
    // cells where there is one tile; the look-back words have room for it)
    k_fill_u32<<<1, 32, 0, st>>>(reinterpret_cast<uint32_t *>(w.ctl), 1, 1u);
    k_scan_lookback<<<1, kScanThreads, 0, st>>>(w.count, w.starts, w.cells, w.ctl, w.err, 0, 1);
    const cudaError_t e = cudaMemsetAsync(w.ctl, 0, 8 * 3, st);
    return e == cudaSuccess ? cudaGetLastError() : e;
}

cudaError_t count_grid_order(cudaStream_t stream, const CountGrid &w, const GridGather *gather) {
    const uint32_t blocks = div_up(w.n, kCountThreads);
    if (gather) k_order<true><<<blocks, kCountThreads, 0, stream>>>(w, *gather);
    else k_order<false><<<blocks, kCountThreads, 0, stream>>>(w, GridGather{});
    return cudaGetLastError();
}

cudaError_t starts_enqueue(cudaStream_t stream, const uint32_t *sorted, uint32_t n, uint32_t cells, uint32_t *starts) {
    // small tiles until the large ones fill the GPU
    if (cells < 148u * kStartMinBlocks * 16u * kStartThreads)
        k_starts<4><<<div_up(cells, 4 * kStartThreads), kStartThreads, 0, stream>>>(sorted, n, cells, starts);
    else
        k_starts<16><<<div_up(cells, 16 * kStartThreads), kStartThreads, 0, stream>>>(sorted, n, cells, starts);
    return cudaGetLastError();
}

cudaError_t grid_build_enqueue(cudaStream_t stream, const float4 *pos, uint32_t n, const GridGeom &g, uint32_t *keys,
                               uint32_t *starts, uint32_t *perm, GridWork &w) {
    cudaError_t e;
    const uint32_t cells = w.cells;
    e = cudaMemsetAsync(w.err, 0, 4 * kErrWords, stream);
    if (e != cudaSuccess) return e;
    if (coop_build_fits(w, stream)) {
        e = coop_build_enqueue(stream, pos, g, keys, starts, perm, w);
        if (e != cudaErrorCooperativeLaunchTooLarge) return e;
    }
    const SortRegion r = sort_region(w.scan_ctl, n, cells, w.passes);
    e = cudaMemsetAsync(w.scan_ctl, 0, w.scan_ctl_bytes, stream);
    if (e != cudaSuccess) return e;
    const uint32_t *sorted = nullptr;
    if (n > 0) {
        const uint32_t blocks = std::min(div_up(n, kSortThreads * kKeyItems), kKeyBlocks);
        k_cell_keys<<<blocks, kSortThreads, 0, stream>>>(pos, n, g, keys, w.passes, r.digit_counts);
        const uint32_t tiles = div_up(n, kSortTile);
        const uint32_t *kin = keys;
        const uint32_t *vin = nullptr;
        for (int pass = 0; pass < w.passes; ++pass) {
            const bool last = pass == w.passes - 1;
            uint32_t *kout = (pass & 1) ? w.k2 : w.k1;
            uint32_t *vout = last ? perm : ((pass & 1) ? w.v2 : w.v1);
            k_radix_pass<<<tiles, kSortThreads, 0, stream>>>(
                kin, vin, n, pass * kRadixBits, r.digit_counts + pass * kRadix, r.tile_status[pass],
                r.tile_ctr[pass], w.err, kout, vout);
            kin = kout;
            vin = vout;
        }
        sorted = kin;
    }
    return starts_enqueue(stream, sorted, n, cells, starts);
}

int32_t report_error(int32_t code, const std::string &msg);

}  // namespace fcu

// The look-back scan's bounded wait, run out on purpose: one block of the
// scan claims tile 1 (the tile counter starts at 1) over a status array in
// which tile 0 never publishes, so its look-back polls status[0] until the
// kSpinLimit bound, records ERRF_SCAN_TIMEOUT and treats the missing prefix
// as zero. Nothing faults or hangs; the context stays usable.
namespace fcu {

int32_t read_build_status(const uint32_t *err, cudaStream_t st, const char *who) {
    uint32_t flags = 0;
    cudaError_t e = cudaMemcpyAsync(&flags, err, 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return report_error(FLUID_ERR_CUDA, std::string(who) + ": " + cudaGetErrorString(e));
    if (flags & (ERRF_SCAN_TIMEOUT | ERRF_SORT_TIMEOUT))
        return report_error(FLUID_ERR_TIMEOUT,
                            std::string(who) + ": a bounded wait of the build gave up; its starts and "
                                               "permutation are invalid");
    return FLUID_OK;
}

cudaError_t enqueue_stalled_radix_pass(const GridWork &w, cudaStream_t st) {
    if (w.n < 2 * kSortTile || w.passes < 1) return cudaErrorInvalidValue;
    const SortRegion r = sort_region(w.scan_ctl, w.n, w.cells, w.passes);
    cudaError_t e = cudaMemsetAsync(w.scan_ctl, 0, w.scan_ctl_bytes, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(w.k2, 0, 4ull * w.n, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(w.err, 0, 4, st);
    if (e != cudaSuccess) return e;
    // the tile counter starts at 1, so the one block claims tile 1
    k_fill_u32<<<1, 32, 0, st>>>(r.tile_ctr[0], 1, 1u);
    k_radix_pass<<<1, kSortThreads, 0, st>>>(w.k2, nullptr, w.n, 0, r.digit_counts, r.tile_status[0],
                                             r.tile_ctr[0], w.err, w.k1, w.v1);
    return cudaGetLastError();
}

}  // namespace fcu

extern "C" int32_t fluid_grid_build_status(const void *workspace, uint32_t n, const FluidGrid *grid,
                                           void *stream) {
    using namespace fcu;
    if (!grid || !workspace) return report_error(FLUID_ERR_ARG, "fluid_grid_build_status: null argument");
    const uint64_t cells = (uint64_t)grid->dims[0] * grid->dims[1] * grid->dims[2];
    if (cells == 0 || cells >= 0xffffffffull)
        return report_error(FLUID_ERR_ARG, "fluid_grid_build_status: bad grid dims");
    const GridWork w = grid_work_carve(const_cast<void *>(workspace), n, (uint32_t)cells, nullptr);
    return read_build_status(w.err, (cudaStream_t)stream, "fluid_grid_build_status");
}

// The bounded look-back wait of a radix digit pass, run out on purpose on a
// real build workspace and reported through fluid_grid_build_status, the
// query a device-pointer caller uses: one block claims tile 1 while tile 0
// never publishes its digit counts, so every digit's look-back gives up. The
// keys are all zero, so the give-up offsets still land inside the outputs.
extern "C" int32_t fluid_selftest_radix_wait(int32_t device, float *ms) {
    using namespace fcu;
    auto fail = [](cudaError_t e) {
        return report_error(FLUID_ERR_CUDA, std::string("fluid_selftest_radix_wait: ") + cudaGetErrorString(e));
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(e);
    const uint32_t n = 2 * kSortTile;
    FluidGrid g{};
    g.cell = 1.0f;
    g.dims[0] = 16;
    g.dims[1] = 16;
    g.dims[2] = 1;
    const size_t bytes = grid_work_bytes(n, 256u);
    void *ws = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    float t = 0.0f;
    int32_t rc = FLUID_OK;
    do {
        if ((e = cudaMalloc(&ws, bytes)) != cudaSuccess) break;
        if ((e = cudaEventCreate(&ev[0])) != cudaSuccess) break;
        if ((e = cudaEventCreate(&ev[1])) != cudaSuccess) break;
        const GridWork w = grid_work_carve(ws, n, 256u, nullptr);
        cudaEventRecord(ev[0]);
        if ((e = enqueue_stalled_radix_pass(w, nullptr)) != cudaSuccess) break;
        cudaEventRecord(ev[1]);
        if ((e = cudaEventSynchronize(ev[1])) != cudaSuccess) break;
        cudaEventElapsedTime(&t, ev[0], ev[1]);
        rc = fluid_grid_build_status(ws, n, &g, nullptr);
    } while (false);
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    cudaFree(ws);
    if (e != cudaSuccess) return fail(e);
    if (ms) *ms = t;
    if (rc == FLUID_ERR_TIMEOUT)
        return report_error(FLUID_ERR_TIMEOUT,
                            "fluid_selftest_radix_wait: the digit look-back wait gave up, as it should, "
                            "and fluid_grid_build_status reported it");
    return rc;
}

extern "C" int32_t fluid_selftest_scan_wait(int32_t device, float *ms) {
    using namespace fcu;
    auto fail = [](cudaError_t e) {
        return report_error(FLUID_ERR_CUDA, std::string("fluid_selftest_scan_wait: ") + cudaGetErrorString(e));
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(e);
    const uint32_t n = 2 * kScanTile;
    uint32_t *in = nullptr, *out = nullptr, *err = nullptr;
    unsigned long long *ctl = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    uint32_t flags = 0;
    float t = 0.0f;
    const unsigned long long one = 1ull;
    do {
        if ((e = cudaMalloc(&in, 4ull * n)) != cudaSuccess) break;
        if ((e = cudaMalloc(&out, 4ull * (n + 1))) != cudaSuccess) break;
        if ((e = cudaMalloc(&ctl, 8ull * 4)) != cudaSuccess) break;
        if ((e = cudaMalloc(&err, 4)) != cudaSuccess) break;
        if ((e = cudaMemset(in, 0, 4ull * n)) != cudaSuccess) break;
        if ((e = cudaMemset(ctl, 0, 8ull * 4)) != cudaSuccess) break;
        if ((e = cudaMemset(err, 0, 4)) != cudaSuccess) break;
        if ((e = cudaMemcpy(ctl, &one, 8, cudaMemcpyHostToDevice)) != cudaSuccess) break;
        if ((e = cudaEventCreate(&ev[0])) != cudaSuccess) break;
        if ((e = cudaEventCreate(&ev[1])) != cudaSuccess) break;
        cudaEventRecord(ev[0]);
        k_scan_lookback<<<1, kScanThreads>>>(in, out, n, ctl, err, 0, 0);
        cudaEventRecord(ev[1]);
        if ((e = cudaEventSynchronize(ev[1])) != cudaSuccess) break;
        if ((e = cudaGetLastError()) != cudaSuccess) break;
        cudaEventElapsedTime(&t, ev[0], ev[1]);
        if ((e = cudaMemcpy(&flags, err, 4, cudaMemcpyDeviceToHost)) != cudaSuccess) break;
    } while (false);
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    cudaFree(in);
    cudaFree(out);
    cudaFree(ctl);
    cudaFree(err);
    if (e != cudaSuccess) return fail(e);
    if (ms) *ms = t;
    if (flags & ERRF_SCAN_TIMEOUT)
        return report_error(FLUID_ERR_TIMEOUT, "fluid_selftest_scan_wait: the look-back wait gave up, as it should");
    return FLUID_OK;
}
