"""The pieces of the cells that the cooperative grid build's blocks write the
starts of: for every accepted cell count, up to 2^32 - 2, the blocks' pieces
are all the cells, each once and in order, and a thread's offset into a piece
never wraps. On the CPU, from the header the kernel includes.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = """
#include <cstdio>
#include <cstdlib>
#include "cell_range.h"
int main(int, char **v) {
    const uint32_t cells = strtoul(v[1], 0, 10), blocks = strtoul(v[2], 0, 10);
    const uint32_t share = fcu::cell_share(cells, blocks);
    for (uint32_t b = 0; b < blocks; ++b) {
        const fcu::CellRange r = fcu::cell_range(cells, share, b);
        printf("%u %u\\n", r.first, r.count);
    }
}
"""


@pytest.fixture(scope="module")
def ranges(tmp_path_factory):
    d = tmp_path_factory.mktemp("cell_range")
    (d / "main.cpp").write_text(MAIN)
    csrc = os.path.join(ROOT, "fluid-simulation-app_b200", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", csrc, "-o", str(d / "main"), str(d / "main.cpp")], check=True)

    def of(cells, blocks):
        out = subprocess.run([str(d / "main"), str(cells), str(blocks)], check=True, capture_output=True, text=True)
        return [tuple(map(int, line.split())) for line in out.stdout.splitlines()]

    return of


@pytest.mark.parametrize("cells", [1, 147, 149, 4096, 151553, 2**31 - 1, 2**31 + 1, 2**32 - 1025, 2**32 - 1024,
                                   2**32 - 1023, 2**32 - 149, 2**32 - 148, 2**32 - 147, 2**32 - 2])
@pytest.mark.parametrize("blocks", [1, 7, 148])
def test_the_blocks_cover_every_cell_once(ranges, cells, blocks):
    if blocks < 148 and -(-cells // 4096) > blocks:
        blocks = 148  # a block never holds more than 4,096 cells unless there is a block per SM
    at = 0
    for first, count in ranges(cells, blocks):
        assert first == at
        at += count
        assert count + 1024 < 2**32
    assert at == cells
