// cell_range.h — the cells whose starts one block of the cooperative grid
// build writes. Plain C++, so that the arithmetic is also checked on the CPU.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define FCU_HD __host__ __device__
#else
#define FCU_HD
#endif

namespace fcu {

struct CellRange {
    uint32_t first, count;
};
// Cells of one of `blocks` even pieces, in 64 bits, since cells + blocks
// passes 2^32 at the largest cell counts. (Once a build, on the host: the
// division in the kernel cost a build of 65,536 positions 0.8 of 23 us.)
FCU_HD inline uint32_t cell_share(uint32_t cells, uint32_t blocks) {
    return (uint32_t)(((uint64_t)cells + blocks - 1) / blocks);
}
// Block b's part of 0 .. cells - 1 in pieces of `share`. first + count never
// passes 2^32, nor does an offset below count that has one stride of a block
// added.
FCU_HD inline CellRange cell_range(uint32_t cells, uint32_t share, uint32_t b) {
    const uint64_t at = (uint64_t)share * b;
    const uint32_t first = at < cells ? (uint32_t)at : cells;
    const uint32_t left = cells - first;
    return CellRange{first, share < left ? share : left};
}

}  // namespace fcu
