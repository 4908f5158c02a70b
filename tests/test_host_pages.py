"""populate_pages (csrc/host_pages.cuh), compiled for the host: it makes fresh
pages present, and changes no byte of pages that hold data, so that a copy
that fails after it leaves the caller's array as it was; memory that cannot be
written is left alone."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mrmd_gb300", "csrc")

DRIVER = r"""
#include "host_pages.cuh"
#include <cstdio>
#include <cstring>
#include <vector>
using namespace mrmd_impl;
int main()
{
    const std::size_t page = (std::size_t)sysconf(_SC_PAGESIZE), n = 64 * page;
    auto map = [&](int prot) {
        return static_cast<unsigned char*>(mmap(nullptr, n, prot, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    };
    auto present = [&](unsigned char* p) {
        std::vector<unsigned char> in(64);
        if (mincore(p, n, in.data()) != 0) return -1;
        int k = 0;
        for (unsigned char c : in) k += c & 1;
        return k;
    };
    // data stays, from any offset and to any length
    unsigned char* a = map(PROT_READ | PROT_WRITE);
    for (std::size_t i = 0; i < n; ++i) a[i] = (unsigned char)(i * 31 + 7);
    populate_pages(a, n);
    populate_pages(a + 8, n - 16);
    populate_pages(a + page - 8, 16);
    for (std::size_t i = 0; i < n; ++i)
        if (a[i] != (unsigned char)(i * 31 + 7)) return std::printf("byte %zu changed\n", i), 1;
    // memory that cannot be written, none at all
    unsigned char* r = map(PROT_READ);
    populate_pages(r, n);
    populate_pages(nullptr, n);
    populate_pages(a, 0);
    // fresh pages, the first and the last of them touched in part
    unsigned char* f = map(PROT_READ | PROT_WRITE);
    populate_pages(f + page - 24, n - 2 * page + 48);
    unsigned char* probe = map(PROT_READ | PROT_WRITE);
    if (madvise(probe, n, MADV_POPULATE_WRITE) != 0) return std::printf("unsupported\n"), 0;
    if (present(f) != 64) return std::printf("%d of 64 pages present\n", present(f)), 1;
    std::printf("ok\n");
}
"""


def test_populate_pages_keeps_data(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    src = tmp_path / "driver.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "driver"
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    if "unsupported" in r.stdout:
        pytest.skip("the kernel has no MADV_POPULATE_WRITE")
