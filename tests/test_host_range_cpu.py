"""Address questions of the host-buffer entry point, compiled for the host and asked of made-up allocations."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "host_range.h"
static const struct { uintptr_t start; size_t size; } kAlloc[] = {{4096, 4096}, {12288, 4096}, {16384, 8192}};   // a hole at 8192, none at 16384
static bool query(uintptr_t p, uintptr_t* start, size_t* size) {
    for (const auto& a : kAlloc)
        if (p >= a.start && p < a.start + a.size) return *start = a.start, *size = a.size, true;
    return false;
}
int main() {
    unsigned long long p, n;
    while (scanf("%llu %llu", &p, &n) == 2) printf("%d\n", (int)b200::inside_one_allocation(query, (uintptr_t)p, (size_t)n));
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_range")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "crispasr_b200", "csrc"), str(d / "main.cpp"), "-o", str(d / "main")],
                   check=True)

    def run(p, n):
        return subprocess.run([str(d / "main")], input=f"{p} {n}", capture_output=True, text=True, check=True).stdout.strip() == "1"
    return run


@pytest.mark.parametrize("p,n,inside", [(4096, 4096, True), (5000, 3192, True), (5000, 3193, False), (4096, 12288, False),   # both ends pinned, a hole between
                                        (8000, 5000, False), (12288, 12288, False), (9000, 10, False), (16384, 8192, True), (24575, 1, True),
                                        (24575, 2, False), (4096, 2 ** 63, False), (4096, 2 ** 64 - 4096, False)])
def test_a_result_is_written_directly_only_inside_one_allocation(ask, p, n, inside):
    """The kernels write a pinned result themselves: every byte of it has to belong to the one allocation that was asked about
    (the ends alone may lie in two, with memory between them that no kernel may touch)."""
    assert ask(p, n) is inside
