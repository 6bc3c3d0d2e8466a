// grid_coop.cu — the neighbour grid of a small or middling input in one
// cooperative launch.
//
// The digit passes of grid.cu are a launch each, with a look-back chain over
// the tiles in every one: up to a million positions that is latency, not
// work (82 us at 1M positions, 39 us at 20k). Here the whole build is one
// kernel of at most a block per SM, each block owning a contiguous piece of
// the input: keys, then per digit the piece ranked (its counts published), a
// grid barrier, the piece's digit offsets from everybody's counts, the piece
// written in digit order through shared memory, a barrier; finally the
// starts, each block searching its share of the cells in the sorted keys, or
// where the cells are many (kStartsApart) k_starts in a launch of its own. A
// digit is as narrow as the keys allow in the same number of passes. The same
// stable order and starts as the digit passes, whatever the distribution.
//
// Barriers are bounded like every wait of the grid: one that gives up sets
// the build's error word, and the writes after it stay in bounds.
//
// Measured, us a build against the digit passes: 20k positions over 14k cells
// 23 / 39, 65k over 33k 23 / 39, 150k over 125k 35 / 56, 400k over 262k 41 /
// 60, 1M over 1M 58 / 82 (in 8 clusters 68 / 91, all in one cell 56 / 70). At
// 1M a pass takes about 13 us, a third of it the two barriers; past one piece a
// block the passes' tiles overlap better (an earlier form at two tiles a block,
// 3M positions: 229, the digit passes of the time 187).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <string>
#include <vector>

#include "cell_range.h"
#include "grid.cuh"

namespace fcu {

int32_t report_error(int32_t code, const std::string &msg);

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;
constexpr uint32_t kTile = kThreads * kItems;  // the largest piece
constexpr int kMinBits = 4, kMaxBits = 8;
constexpr uint32_t kMaxDigits = 1u << kMaxBits;

struct Coop {
    const float4 *pos;
    GridGeom g;
    uint32_t n, cells, blocks, piece, share;  // piece, share: positions and cells a block owns
    int passes, bits;          // digit passes of `bits` bits each
    uint2 *a, *b;              // (key, index) ping-pong
    uint32_t *keys;            // the caller's keys, or null
    uint32_t *starts, *perm;   // starts null: not written here
    uint32_t *counts;          // [block][digit]
    uint32_t *barrier, *err;
};

struct CoopShared {
    uint32_t hist[kWarps][kMaxDigits];
    uint2 pair[kTile];
    uint32_t off[kMaxDigits], start[kMaxDigits];  // output and staged index of a digit's first element
    uint32_t part[4][kMaxDigits], before[4][kMaxDigits];
    uint32_t sum[kWarps];
    uint32_t lo, hi;
};

// Every block's `phase`-th arrival.
__device__ void grid_barrier(const Coop &c, uint32_t phase) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(c.barrier, 1u);
        const uint32_t want = phase * gridDim.x;
        uint32_t v, spins = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(c.barrier) : "memory");
        } while (v < want && ++spins < kSpinLimit);
        if (v < want) atomicOr(c.err, ERRF_SORT_TIMEOUT);
        __threadfence();
    }
    __syncthreads();
}

__device__ __forceinline__ uint2 ld_pair(const uint2 *p) { return __ldcg(p); }  // other blocks wrote it

// Exclusive scan over the digits of the first kMaxDigits threads' values, in
// two halves around a __syncthreads.
__device__ __forceinline__ uint32_t digit_scan_warp(CoopShared &s, uint32_t v) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s.sum[warp] = x;
    return x - v;
}
__device__ __forceinline__ uint32_t digit_scan_block(const CoopShared &s) {
    uint32_t w = 0;
#pragma unroll
    for (uint32_t k = 0; k < kMaxDigits / 32; ++k)
        if (k < threadIdx.x >> 5) w += s.sum[k];
    return w;
}

template <int kBits>
__global__ void __launch_bounds__(kThreads, 1) k_grid_coop(Coop c) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    CoopShared &s = *reinterpret_cast<CoopShared *>(s_raw);
    constexpr uint32_t kDigits = 1u << kBits, kMask = kDigits - 1u;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t first = min(blockIdx.x * c.piece, c.n), len = min(c.piece, c.n - first);
    // warp w holds a contiguous run of the piece, so that ranks taken round
    // by round keep the input order
    const int rounds = (int)((len + kThreads - 1) / kThreads);
    const uint32_t run = warp * 32u * rounds;
    uint32_t phase = 0;

    for (uint32_t i = first + tid; i < first + len; i += kThreads) {
        const float4 p = __ldg(&c.pos[i]);
        const uint32_t cx = axis_cell(p.x, c.g.min[0], c.g.cell, c.g.dims[0]);
        const uint32_t cy = axis_cell(p.y, c.g.min[1], c.g.cell, c.g.dims[1]);
        const uint32_t cz = axis_cell(p.z, c.g.min[2], c.g.cell, c.g.dims[2]);
        const uint32_t key = (cz * c.g.dims[1] + cy) * c.g.dims[0] + cx;
        c.a[i] = make_uint2(key, i);  // read back by this block alone
        if (c.keys) c.keys[i] = key;
    }
    __syncthreads();

    const uint2 *in = c.a;
    uint2 *out = c.b;
    for (int pass = 0; pass < c.passes; ++pass) {
        const bool last = pass == c.passes - 1;
        const int shift = pass * kBits;
        uint2 p[kItems];
        uint32_t rank[kItems];
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const uint32_t q = run + r * 32 + lane;
            p[r] = r < rounds && q < len ? ld_pair(&in[first + q]) : make_uint2(0u, 0u);
        }
        for (uint32_t d = lane; d < kMaxDigits; d += 32) s.hist[warp][d] = 0u;
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            if (r >= rounds) break;
            const bool live = run + r * 32 + lane < len;
            const uint32_t d = (p[r].x >> shift) & kMask;
            uint32_t peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
            for (int b = 0; b < kBits; ++b) {
                const uint32_t bit = (d >> b) & 1u, bal = __ballot_sync(0xffffffffu, bit);
                peers &= bit ? bal : ~bal;
            }
            uint32_t before = 0;
            const uint32_t leader = live ? (uint32_t)__ffs(peers) - 1u : lane;
            if (live && lane == leader) {
                before = s.hist[warp][d];
                s.hist[warp][d] = before + (uint32_t)__popc(peers);
            }
            rank[r] = __shfl_sync(0xffffffffu, before, leader) + __popc(peers & ((1u << lane) - 1u));
            __syncwarp();
        }
        __syncthreads();
        // the warps' exclusive counts of a digit, the piece's count of it for
        // the other blocks, and the digits' staged starts
        uint32_t mine = 0;
        if (tid < kMaxDigits) {
            uint32_t total = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t v = s.hist[w][tid];
                s.hist[w][tid] = total;
                total += v;
            }
            if (tid < kDigits) c.counts[blockIdx.x * kDigits + tid] = total;
            mine = digit_scan_warp(s, total);
        }
        __syncthreads();
        if (tid < kMaxDigits) s.start[tid] = mine + digit_scan_block(s);
        __syncthreads();
        // staged while the barrier waits for the other blocks
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            if (r >= rounds) break;
            if (run + r * 32 + lane < len) {
                const uint32_t d = (p[r].x >> shift) & kMask;
                s.pair[s.start[d] + s.hist[warp][d] + rank[r]] = p[r];
            }
        }
        grid_barrier(c, ++phase);

        // offsets: the digit's elements in earlier pieces, and all smaller
        // digits' elements; four groups of threads share the pieces
        {
            const uint32_t d = tid % kMaxDigits, q = tid / kMaxDigits;
            uint32_t all = 0, pre = 0;
            if (d < kDigits) {
#pragma unroll 8
                for (uint32_t b = q; b < gridDim.x; b += 4) {
                    const uint32_t v = __ldcg(&c.counts[b * kDigits + d]);
                    all += v;
                    if (b < blockIdx.x) pre += v;
                }
            }
            s.part[q][d] = all;
            s.before[q][d] = pre;
        }
        __syncthreads();
        if (tid < kMaxDigits)
            mine = digit_scan_warp(s, s.part[0][tid] + s.part[1][tid] + s.part[2][tid] + s.part[3][tid]);
        __syncthreads();
        if (tid < kMaxDigits)
            s.off[tid] = mine + digit_scan_block(s) + s.before[0][tid] + s.before[1][tid] + s.before[2][tid] +
                         s.before[3][tid];
        __syncthreads();
        for (uint32_t j = tid; j < len; j += kThreads) {
            const uint2 v = s.pair[j];
            const uint32_t d = (v.x >> shift) & kMask;
            const uint32_t dst = s.off[d] + (j - s.start[d]);
            if (dst >= c.n) continue;  // only after a barrier that gave up
            if (last) {
                c.perm[dst] = v.y;
                reinterpret_cast<uint32_t *>(out)[dst] = v.x;
            } else {
                out[dst] = v;
            }
        }
        if (last && !c.starts) return;  // the starts have a launch of their own
        grid_barrier(c, ++phase);
        uint2 *const was = const_cast<uint2 *>(in);
        in = out;
        out = was;
    }

    // starts: this block's share of the cells in the sorted keys
    const uint32_t *sorted = reinterpret_cast<const uint32_t *>(in);
    const CellRange r = cell_range(c.cells, c.share, blockIdx.x);
    if (warp < 2) {
        const uint32_t at = warp_lower_bound(sorted, c.n, warp ? r.first + r.count : r.first);
        if (lane == 0) (warp ? s.hi : s.lo) = at;
    }
    __syncthreads();
    const uint32_t lo = s.lo, m = s.hi > lo ? s.hi - lo : 0u;
    uint32_t *k = reinterpret_cast<uint32_t *>(s.pair);
    const bool staged = m <= 2 * kTile;
    if (staged)
        for (uint32_t j = tid; j < m; j += kThreads) k[j] = __ldcg(&sorted[lo + j]);
    __syncthreads();
    for (uint32_t x = tid; x < r.count; x += kThreads) {
        const uint32_t cell = r.first + x;
        uint32_t at = 0, top = m;
        while (at < top) {
            const uint32_t mid = (at + top) >> 1;
            const uint32_t v = staged ? k[mid] : __ldcg(&sorted[lo + mid]);
            if (v < cell) at = mid + 1;
            else top = mid;
        }
        c.starts[cell] = lo + at;
    }
    if (blockIdx.x == 0 && tid == 0) c.starts[c.cells] = c.n;
}

// Passes, digit width and pieces: a block per SM where the positions or the
// cells (their starts) are many.
Coop shape_of(const GridWork &w) {
    Coop c{};
    c.n = w.n;
    c.cells = w.cells;
    int bits = 0;
    while (bits < 32 && ((uint64_t)w.cells - 1) >> bits) ++bits;
    c.passes = std::max(1, (bits + kMaxBits - 1) / kMaxBits);
    c.bits = std::max(kMinBits, (bits + c.passes - 1) / c.passes);
    c.blocks = std::min(kCoopBlocks, std::max(div_up(w.n, kThreads), div_up(w.cells, 4096u)));
    c.piece = std::max((uint32_t)kThreads, div_up(div_up(w.n, c.blocks), 32) * 32);
    c.share = cell_share(w.cells, c.blocks);
    return c;
}

template <int kBits>
cudaError_t launch(cudaStream_t stream, Coop &c) {
    if (c.bits != kBits) {
        if constexpr (kBits > kMinBits) return launch<kBits - 1>(stream, c);
    }
    const cudaError_t e = cudaFuncSetAttribute(k_grid_coop<kBits>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(CoopShared));
    if (e != cudaSuccess) return e;
    void *args[] = {&c};
    const cudaError_t l = cudaLaunchCooperativeKernel((const void *)k_grid_coop<kBits>, dim3(c.blocks), dim3(kThreads),
                                                      args, sizeof(CoopShared), stream);
    if (l == cudaErrorCooperativeLaunchTooLarge) (void)cudaGetLastError();  // the caller goes another way
    return l;
}

// Cells from which the starts are k_starts' launch after this one: a thread
// here searches a cell's start among its block's keys, which past some
// thousand cells a block costs more than a launch that reads the keys once. us
// a build with the starts here / apart / by digit passes, 1M positions, in any
// order and all in one cell: 262k cells 53 / 54 / 78 and 54 / 52 / 68, 512k 58
// / 56 / 79 and 64 / 54 / 69, 1M 62 / 58 / 82 and 75 / 56 / 70, 4.1M 94 / 63 /
// 84 and 154 / 64 / 74, 16.8M 211 / 81 / 101 and 463 / 77 / 88; 150k positions
// over 262k cells 35 / 35 / 56, over 2.1M 50 / 42 / 62.
constexpr uint32_t kStartsApart = 400000;
bool starts_apart(const GridWork &w) { return w.cells > kStartsApart; }

// Driver entry points, null where the driver has none.
struct SmCalls {
    PFN_cuStreamGetGreenCtx ctx_of = nullptr;
    PFN_cuGreenCtxGetDevResource of_green = nullptr;
    PFN_cuCtxGetCurrent current = nullptr;
    PFN_cuCtxGetDevResource of_ctx = nullptr;
};
const SmCalls &sm_calls() {
    static const SmCalls calls = [] {
        SmCalls c;
        void *p[4] = {nullptr, nullptr, nullptr, nullptr};
        const char *const name[4] = {"cuStreamGetGreenCtx", "cuGreenCtxGetDevResource", "cuCtxGetCurrent",
                                     "cuCtxGetDevResource"};
        for (int k = 0; k < 4; ++k) {
            cudaDriverEntryPointQueryResult found;
            if (cudaGetDriverEntryPointByVersion(name[k], &p[k], 12040, cudaEnableDefault, &found) != cudaSuccess ||
                found != cudaDriverEntryPointSuccess)
                return c;
        }
        c.ctx_of = reinterpret_cast<PFN_cuStreamGetGreenCtx>(p[0]);
        c.of_green = reinterpret_cast<PFN_cuGreenCtxGetDevResource>(p[1]);
        c.current = reinterpret_cast<PFN_cuCtxGetCurrent>(p[2]);
        c.of_ctx = reinterpret_cast<PFN_cuCtxGetDevResource>(p[3]);
        return c;
    }();
    return calls;
}

// SMs the stream's kernels may run on: its green context's, for a default
// stream the current context's (which may be a green one's), else the device's.
uint32_t sms_of(cudaStream_t stream) {
    const SmCalls &calls = sm_calls();
    CUdevResource r{};
    if (calls.ctx_of) {
        CUgreenCtx green = nullptr;
        if (stream == nullptr || stream == cudaStreamLegacy || stream == cudaStreamPerThread) {
            CUcontext ctx = nullptr;
            if (calls.current(&ctx) == CUDA_SUCCESS && ctx &&
                calls.of_ctx(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS)
                return r.sm.smCount;
        } else if (calls.ctx_of(stream, &green) == CUDA_SUCCESS && green) {
            return calls.of_green(green, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS ? r.sm.smCount : 0u;
        }
    }
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0u;
    return (uint32_t)sms;
}

}  // namespace

bool coop_build_fits(const GridWork &w, cudaStream_t stream) {
    if (w.n == 0 || w.n > kCoopBlocks * kTile) return false;
    const Coop c = shape_of(w);
    // every block resident at once: a stream with fewer SMs to give (a slice
    // of the device, a green context) builds by digit passes
    if (sms_of(stream) < c.blocks) return false;
    return 4ull * ((uint64_t)c.blocks << c.bits) <= w.scan_ctl_bytes;
}

cudaError_t coop_build_enqueue(cudaStream_t stream, const float4 *pos, const GridGeom &g, uint32_t *keys,
                               uint32_t *starts, uint32_t *perm, const GridWork &w) {
    Coop c = shape_of(w);
    c.pos = pos;
    c.g = g;
    c.a = reinterpret_cast<uint2 *>(w.k1);       // k1, k2
    c.b = reinterpret_cast<uint2 *>(w.v1);       // v1, v2
    c.keys = keys == w.k2 ? nullptr : keys;      // k2: no buffer of the caller's
    const bool apart = starts_apart(w);
    c.starts = apart ? nullptr : starts;
    c.perm = perm;
    c.counts = reinterpret_cast<uint32_t *>(w.scan_ctl);
    c.err = w.err;
    c.barrier = w.err + kErrBarrier;
    const cudaError_t e = launch<kMaxBits>(stream, c);
    if (e != cudaSuccess || !apart) return e;
    // the last pass left the sorted keys in its output
    return starts_enqueue(stream, c.passes & 1 ? w.v1 : w.k1, w.n, w.cells, starts);
}

cudaError_t enqueue_stalled_coop_build(cudaStream_t stream, const float4 *pos, const GridGeom &g, uint32_t *starts,
                                       uint32_t *perm, const GridWork &w) {
    if (!coop_build_fits(w, stream)) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(w.err, 0, 4 * kErrWords, stream);
    // one arrival short from the first barrier on: its count starts at -1
    if (e == cudaSuccess) e = cudaMemsetAsync(w.err + kErrBarrier, 0xff, 4, stream);
    if (e == cudaSuccess) e = coop_build_enqueue(stream, pos, g, w.k2, starts, perm, w);
    return e;
}

}  // namespace fcu

// The build's barrier, run out on purpose on a real workspace and reported
// through fluid_grid_build_status: every barrier expects an arrival more than
// come, so every block gives up at every one and the kernel ends by itself.
// What it then writes from counts that nobody published stays inside the
// outputs: the words on either side of them are checked.
extern "C" int32_t fluid_selftest_coop_wait(int32_t device, float *ms) {
    using namespace fcu;
    auto fail = [](cudaError_t e) {
        return report_error(FLUID_ERR_CUDA, std::string("fluid_selftest_coop_wait: ") + cudaGetErrorString(e));
    };
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return fail(e);
    constexpr uint32_t n = 5003, side = 16, cells = side * side * side, guard = 64, mark = 0xa5a5a5a5u;
    FluidGrid grid{};
    grid.cell = 1.0f;
    for (int a = 0; a < 3; ++a) grid.dims[a] = side;
    GridGeom g{};
    g.cell = 1.0f;
    for (int a = 0; a < 3; ++a) g.dims[a] = side;
    const size_t words = 3 * guard + cells + 1 + n;  // guard, starts, guard, perm, guard
    std::vector<uint32_t> out(words, 0u);
    std::vector<float> at(4 * n);
    for (size_t k = 0; k < at.size(); ++k) at[k] = (float)((k * 7919u) % 1600u) * 0.01f;
    char *ws = nullptr;
    uint32_t *dst = nullptr;
    float4 *pos = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    float t = 0.0f;
    int32_t rc = FLUID_OK;
    do {
        const size_t bytes = grid_work_bytes(n, cells);
        if ((e = cudaMalloc(&ws, bytes)) != cudaSuccess) break;
        if ((e = cudaMalloc(&dst, 4 * words)) != cudaSuccess) break;
        if ((e = cudaMalloc(&pos, 16 * n)) != cudaSuccess) break;
        if ((e = cudaMemset(ws, 0x5a, bytes)) != cudaSuccess) break;
        if ((e = cudaMemset(dst, 0xa5, 4 * words)) != cudaSuccess) break;
        if ((e = cudaMemcpy(pos, at.data(), 16 * n, cudaMemcpyHostToDevice)) != cudaSuccess) break;
        if ((e = cudaEventCreate(&ev[0])) != cudaSuccess) break;
        if ((e = cudaEventCreate(&ev[1])) != cudaSuccess) break;
        const GridWork w = grid_work_carve(ws, n, cells, nullptr);
        cudaEventRecord(ev[0]);
        e = enqueue_stalled_coop_build(nullptr, pos, g, dst + guard, dst + 2 * guard + cells + 1, w);
        if (e != cudaSuccess) break;
        cudaEventRecord(ev[1]);
        if ((e = cudaEventSynchronize(ev[1])) != cudaSuccess) break;
        cudaEventElapsedTime(&t, ev[0], ev[1]);
        rc = fluid_grid_build_status(ws, n, &grid, nullptr);
        if ((e = cudaMemcpy(out.data(), dst, 4 * words, cudaMemcpyDeviceToHost)) != cudaSuccess) break;
    } while (false);
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    cudaFree(ws);
    cudaFree(dst);
    cudaFree(pos);
    if (e != cudaSuccess) return fail(e);
    if (ms) *ms = t;
    for (size_t k = 0; k < guard; ++k)
        if (out[k] != mark || out[guard + cells + 1 + k] != mark || out[words - 1 - k] != mark)
            return report_error(FLUID_ERR_STATE, "fluid_selftest_coop_wait: a write outside the outputs");
    if (rc == FLUID_ERR_TIMEOUT)
        return report_error(FLUID_ERR_TIMEOUT,
                            "fluid_selftest_coop_wait: the grid barrier gave up, as it should, and "
                            "fluid_grid_build_status reported it");
    return rc;
}
