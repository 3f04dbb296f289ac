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
int main(int argc, char**) {
    unsigned long long a[7];
    if (argc > 1) {
        for (auto& x : a) if (scanf("%llu", &x) != 1) return 1;
        printf("%d\n", (int)b200::result_meets(a[0], a[1], a[2], a[3], a[4], a[5], a[6]));
    } else if (scanf("%llu %llu", &a[0], &a[1]) == 2) {
        printf("%d\n", (int)b200::inside_one_allocation(query, (uintptr_t)a[0], (size_t)a[1]));
    }
}
"""


@pytest.fixture(scope="module")
def ask(tmp_path_factory):
    d = tmp_path_factory.mktemp("host_range")
    (d / "main.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "crispasr_b200", "csrc"), str(d / "main.cpp"), "-o", str(d / "main")],
                   check=True)

    def run(*numbers):
        args = [str(d / "main")] + ["meets"] * (len(numbers) > 2)
        return int(subprocess.run(args, input=" ".join(map(str, numbers)), capture_output=True, text=True, check=True).stdout)
    return run


@pytest.mark.parametrize("p,n,inside", [(4096, 4096, True), (5000, 3192, True), (5000, 3193, False), (4096, 12288, False),   # both ends pinned, a hole between
                                        (8000, 5000, False), (12288, 12288, False), (9000, 10, False), (16384, 8192, True), (24575, 1, True),
                                        (24575, 2, False), (4096, 2 ** 63, False), (4096, 2 ** 64 - 4096, False)])
def test_a_result_is_written_directly_only_inside_one_allocation(ask, p, n, inside):
    """The kernels write a pinned result themselves: every byte of it has to belong to the one allocation that was asked about
    (the ends alone may lie in two, with memory between them that no kernel may touch)."""
    assert bool(ask(p, n)) is inside


# result: 4 entries of 100 bytes at 1000
@pytest.mark.parametrize("p,stride,nbytes,m,meets", [
    (1000, 100, 100, 4, 1),      # the operand itself is updated
    (1020, 100, 60, 4, 1),       # rows inside each entry
    (1020, 100, 90, 4, 2),       # reaches into the next entry
    (1000, 200, 100, 4, 2),      # entries wander
    (1000, 100, 100, 3, 2),      # another number of entries
    (1300, 100, 100, 1, 2),      # a shared operand inside the last entry
    (990, 100, 100, 4, 2),       # starts before
    (1400, 100, 100, 4, 0), (600, 100, 100, 4, 0), (601, 100, 100, 4, 2)])
def test_how_a_result_meets_an_operand(ask, p, stride, nbytes, m, meets):
    """0 apart, 1 entry by entry (an update in place), 2 any other way."""
    assert ask(1000, 100, 4, p, stride, nbytes, m) == meets
