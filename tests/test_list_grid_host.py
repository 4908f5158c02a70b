"""The cells of a list build (csrc/list_grid.cuh), compiled for the host: their
number without wrapping, and half-radius cells only where 31 bits number them,
so that a dilute system of hundreds of millions of particles, whose
full-radius cells can be, keeps its list."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mrmd_gb300", "csrc")

DRIVER = r"""
#include "list_grid.cuh"
#include <cstdio>
using namespace mrmd_impl;
int main()
{
    // counts past 31 bits, and products past 63, do not wrap
    struct { double L, edge; int64_t n; } a[] = {
        {10.0, 3.0, 3}, {2.0, 3.0, 1}, {2147483646.5, 1.0, 2147483646}, {2147483647.0, 1.0, 2147483647},
        {4294967297.0, 1.0, 2147483647}, {1e300, 1e-300, 2147483647}};
    for (auto& k : a)
        if (cells_per_axis(k.L, k.edge) != k.n) return std::printf("%g / %g\n", k.L, k.edge), 1;
    const int64_t M = 2147483647;
    if (cell_count(3, 4, 5) != 60 || cell_count(M, 1, 1) != M || cell_count(M, 9, 1) != 9 * M || cell_count(M, M, 1) <= M ||
        cell_count(M, M, M) <= M)
        return std::printf("cell_count\n"), 1;
    struct { int64_t cells, n; bool half; } c[] = {
        {1, 1, true}, {27, 0, true}, {1048576, 0, true}, {1048577, 0, false}, {1048584, 1, true},
        {1048585, 1, false}, {8 * 256000, 256000, true}, {10000000, 4000, false},
        // 300,000,000 particles: up to 2^31 - 1 cells, whatever the particles allow
        {M, 300000000, true}, {M + 1, 300000000, false}, {2400000000, 300000000, false},
        {4000000000, 2147483647, false}, {(int64_t)1 << 48, 2147483647, false}};
    for (auto& k : c)
        if (half_radius_cells(k.cells, k.n) != k.half)
            return std::printf("%lld cells, %lld particles\n", (long long)k.cells, (long long)k.n), 1;
    return 0;
}
"""


def test_cells_have_31_bit_indices(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "driver"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
