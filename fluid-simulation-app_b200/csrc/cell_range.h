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
// Block b's part of 0 .. cells - 1 in `blocks` even pieces. In 64 bits, since
// cells + blocks passes 2^32 at the largest cell counts; first + count never
// does, nor does an offset below count that has one stride of a block added.
FCU_HD inline CellRange cell_range(uint32_t cells, uint32_t blocks, uint32_t b) {
    const uint64_t share = ((uint64_t)cells + blocks - 1) / blocks;
    const uint64_t at = share * b, first = at < cells ? at : cells;
    const uint64_t left = cells - first;
    return CellRange{(uint32_t)first, (uint32_t)(share < left ? share : left)};
}

}  // namespace fcu
