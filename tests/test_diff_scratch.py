"""The places of the differentiable backward's checkpoints, as the host and the kernel
compute them: tiles do not share one and none lies outside the buffer, also beyond
2^24 chunks (2^32 floats)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "kernels.h"
int main(int argc, char** argv) {  // records per tile, from the tile whose records start at argv[1]
    uint64_t start = strtoull(argv[1], nullptr, 10), tile = strtoull(argv[2], nullptr, 10);
    for (int k = 3; k < argc; ++k) {
        const uint64_t n = strtoull(argv[k], nullptr, 10);
        printf("%llu %llu ", (unsigned long long)tk::diff_scratch_at(start, tile), (unsigned long long)n);
        start += n;
        ++tile;
    }
    printf("%llu\n", (unsigned long long)tk::diff_scratch_len(start, tile));
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("scratch")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "tileink_b200" / "csrc"), "-I", "/usr/local/cuda/include",
                    str(d / "p.cpp"), "-o", str(d / "p")], check=True)
    return d / "p"


# (tile's first record + its number in chunks) below, across and above 2^24 chunks
@pytest.mark.parametrize("start,tile", [(0, 0), (2**28 - 40, 0), (2**28 - 2**20, 2**16 - 3), (2**32 - 4096, 2**20)])
def test_diff_checkpoints_apart(program, start, tile):
    counts = [1, 15, 16, 17, 0, 33, 1, 1, 31, 400]
    out = subprocess.run([str(program), str(start), str(tile), *map(str, counts)], check=True, capture_output=True, text=True)
    v = [int(x) for x in out.stdout.split()]
    end, length = (start // 16 + tile) * 256, v.pop()
    assert v[0] == end
    for at, n in zip(v[::2], v[1::2]):
        assert at >= end
        end = at + 256 * ((n + 15) // 16)
    assert end <= length


def test_diff_kernel_takes_the_shared_place():
    src = (ROOT / "tileink_b200" / "csrc" / "diff.cu").read_text()
    assert "scratch + diff_scratch_at(rec.ptcl_start, tile) + tid" in src
