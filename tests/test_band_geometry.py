"""The tiles of the Coulomb bands (csrc/nd_bands.cuh), compiled for the host:
the rows whose position and charge the term kernel loads exist, and every pair
lies in exactly one tile."""
import os
import subprocess

import pytest

from conftest import PKG

SRC = r"""
#include <stdio.h>
#include <stdlib.h>
#include <vector>
#include "nd_bands.cuh"
using namespace nd;
int main(int argc, char** argv) {
    const int32_t n = atoi(argv[1]), P = band_steps(n), nband = (n + kBandRows - 1) / kBandRows;
    long long cells = 0, bad = 0, twice = 0;
    std::vector<unsigned char> seen((size_t)n * n, 0);
    for (int32_t b = 0; b < nband; ++b)
        for (int32_t t = 0; t < P - 64 * b; ++t)
            for (int32_t lane = 0; lane < 32; ++lane)
                for (int32_t r = 0; r < 8; ++r) {
                    const int32_t i = band_row(b, lane, r), j0 = band_col(b, lane, t);
                    if (!band_tile_has_pair(i, j0, n)) continue;
                    if (i < 0 || i >= n) { ++bad; continue; }  // x[3 i], q[i] are loaded
                    for (int32_t j = j0; j < j0 + 4; ++j)
                        if (j > i && j < n) { ++cells; twice += seen[(size_t)i * n + j]++ != 0; }
                }
    printf("%lld %lld %lld\n", bad, cells, twice);
}
"""


@pytest.fixture(scope="module")
def geometry(tmp_path_factory):
    d = tmp_path_factory.mktemp("bands")
    (d / "g.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(PKG, "csrc"), str(d / "g.cpp"),
                    "-o", str(d / "g")], check=True)
    return str(d / "g")


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 31, 254, 255, 256, 257, 258, 509, 514, 1021, 2046])
def test_rows_exist_and_pairs_once(geometry, n):
    bad, cells, twice = map(int, subprocess.run([geometry, str(n)], capture_output=True, text=True,
                                                check=True).stdout.split())
    assert bad == 0 and twice == 0 and cells == n * (n - 1) // 2
