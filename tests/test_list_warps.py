"""The list builds' warps per key, compiled from the library's header: their number stays
within the kernels' 32-bit indexes for every grid that is accepted, up to 2^29 cells, and
a mostly empty grid gets one warp per key."""
import os
import subprocess
import tempfile

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include <cstdio>
#include <cstdlib>
#include "mph_internal.h"
int main(int argc, char** argv) {
    for (int k = 1; k + 2 < argc; k += 3)
        std::printf("%d\\n", mph::list_key_warps(std::atoi(argv[k]), std::atoi(argv[k + 1]), std::atoi(argv[k + 2])));
    return mph::kListWarps;
}
"""


@pytest.fixture(scope="module")
def key_warps():
    with tempfile.TemporaryDirectory() as td:
        src, exe = os.path.join(td, "a.cpp"), os.path.join(td, "a")
        with open(src, "w") as f:
            f.write(SRC)
        cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
        subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "mphexplicit_b200", "csrc"), "-I",
                        os.path.join(ROOT, "include"), "-I", os.path.join(cuda, "include"), src, "-o", exe], check=True)

        def ask(cases):
            r = subprocess.run([exe] + [str(v) for c in cases for v in c], stdout=subprocess.PIPE, text=True)
            return [int(v) for v in r.stdout.split()], r.returncode

        yield ask


def test_warps_are_numbered_in_32_bits(key_warps):
    cases = [(dim, n, tot) for dim in (2, 3) for n in (1, 50000, 250000, 250001, 10 ** 8)
             for tot in (1, 1 << 16, 1 << 20, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1, 1 << 29)]
    got, per_block = key_warps(cases)
    assert len(got) == len(cases) and per_block > 0
    for (dim, n, tot), w in zip(cases, got):
        assert w >= 1
        blocks = -(-2 * tot * w // per_block)
        assert blocks * per_block - 1 < 2 ** 31, (dim, n, tot, w)  # the last warp's number


def test_empty_keys_get_one_warp(key_warps):
    cases = [(3, 20116, 2000), (3, 213868, 14000), (3, 2779256, 160000), (2, 22500, 1800), (2, 90000, 7000),
             (3, 8000, 1000000), (3, 216000, 4096000), (2, 3600, 90000)]
    assert key_warps(cases)[0] == [4, 4, 2, 2, 1, 1, 1, 1]
