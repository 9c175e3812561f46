"""Mapping the pages of a result buffer ahead of its copy (csrc/host_pages.h)
changes nothing in it: a call that fails later leaves the caller's data as it
was, and a buffer that the CPU may not write is no fault there."""
from __future__ import annotations

import subprocess

from conftest import ROOT

CSRC = ROOT / "lbm_bench_gpu_gb300" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "host_pages.h"

int main()
{
    const size_t page = (size_t)sysconf(_SC_PAGESIZE), n = 40 * page;
    auto map = [&](int prot) { return (unsigned char *)mmap(nullptr, n, prot, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0); };
    const auto never = [] { return false; };
    // a buffer in use, with ragged ends: every byte stays
    std::vector<unsigned char> v(n);
    for (size_t i = 0; i < n; i++) v[i] = (unsigned char)(i * 7 + 3);
    lbm::populate_pages(v.data() + 5, n - 11, never);
    for (size_t i = 0; i < n; i++)
        if (v[i] != (unsigned char)(i * 7 + 3)) return 1;
    // memory that cannot be written, and memory that is not there
    unsigned char *ro = map(PROT_READ), *gone = map(PROT_READ | PROT_WRITE);
    if (ro == MAP_FAILED || gone == MAP_FAILED) return 2;
    munmap(gone, n);
    lbm::populate_pages(ro, n, never);
    lbm::populate_pages(gone, n, never);
    for (size_t i = 0; i < n; i += page)
        if (ro[i] != 0) return 3;
    // untouched memory is mapped (where the kernel has the call), all of it or until done
    unsigned char *a = map(PROT_READ | PROT_WRITE), *b = map(PROT_READ | PROT_WRITE), *c = map(PROT_READ | PROT_WRITE);
    const bool has = madvise(c, page, MADV_POPULATE_WRITE) == 0;
    int asked = 0;
    lbm::populate_pages(a, n, never);
    lbm::populate_pages(b, n, [&] { return asked++ == 2; });
    std::vector<unsigned char> in_a(n / page), in_b(n / page);
    if (mincore(a, n, in_a.data()) || mincore(b, n, in_b.data())) return 4;
    for (size_t i = 0; has && i < n / page; i++)
        if (!(in_a[i] & 1) || (in_b[i] & 1) != (i < 16)) return 5;
    return asked <= 3 ? 0 : 6;
}
"""


def test_populate_changes_no_byte_and_faults_nowhere(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
