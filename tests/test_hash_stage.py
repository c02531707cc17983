"""Sizes of the staged hash-grid insert, compiled on their own for the host."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rtlib_b200", "csrc")

PROGRAM = r"""
#include "hash_stage.h"
#include <stdio.h>
using namespace rtpg;
int main() {
    const uint64_t n[] = {1, 21, 22, 65536, 1ull << 22, 1ull << 30, (1ull << 30) + 1, 1431655765, 1431655766, 1500000000, 1ull << 31,
                          4000000000ull, 0xffffffffull, 1ull << 40};
    const uint64_t slots[] = {32, 1ull << 20, 1ull << 28, 1ull << 29, 0xffffffe0ull};
    for (uint64_t p : n)
        for (uint64_t s : slots) {
            const uint32_t cap = stage_cap(p, s);
            printf("%llu %llu %d %u %u\n", (unsigned long long)p, (unsigned long long)s, (int)stage_fits(p, s), cap, stage_size(cap));
        }
}
"""


def test_stage_sizes_up_to_the_largest_batch(tmp_path):
    """Every staged batch finds a table with free entries, numbered in 32 bits; larger batches are left
    to the sorted insert; no size keeps the doubling from ending."""
    (tmp_path / "p.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "p")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(tmp_path / "p.cpp"), "-o", exe])
    rows = subprocess.run([exe], stdout=subprocess.PIPE, check=True, timeout=60).stdout.decode().split("\n")
    seen = 0
    for row in filter(None, rows):
        points, slots, fits, cap, size = map(int, row.split())
        assert fits == (points <= min(1 << 30, 4 * slots))
        assert cap == min(points, 1 << 30, 4 * slots)  # never more than what fits
        assert size & (size - 1) == 0 and 2 * size >= 3 * cap - 1 and (size == 32 or size < 3 * cap) and size <= 1 << 31
        seen += 1
    assert seen == 70
