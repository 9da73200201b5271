"""The walk of a thread through the items of a grid (Strided) where the items come near 2^32,
the limit of gpe_create: it ends, and the threads' walks together take every item once."""
import os
import re
import subprocess

from spacetime_gb300 import build

PROGRAM = r"""
#include <cstdio>
#include "gpe_internal.h"
int main() {
    // item counts, thread counts: ordinary, and where first + k stride passes 2^32
    const uint32_t totals[] = {1u, 7u, 1000u, 0x7fffffffu, 0x80000000u, 0xffff0000u, 0xfffffff0u, 0xffffffffu};
    const uint32_t strides[] = {1u << 8, 77824u, 311296u, 0x10000000u, 0x80000000u, 0xfffffff0u};
    for (uint32_t total : totals)
        for (uint32_t stride : strides) {
            const uint32_t firsts[] = {0u, 1u, stride / 2, stride - 1u, total - 1u, total};
            for (uint32_t first : firsts) {
                uint64_t steps = 0, at = first;
                const uint64_t want = first < total ? ((uint64_t)total - first + stride - 1) / stride : 0;
                for (gpe::Strided it(first, stride, total); it.more(); it.next(), ++steps, at += stride)
                    if (it.i != at || steps >= want) return std::printf("total %u stride %u first %u step %llu\n", total, stride,
                                                                       first, (unsigned long long)steps), 1;
                if (steps != want) return std::printf("total %u stride %u first %u: %llu of %llu\n", total, stride, first,
                                                      (unsigned long long)steps, (unsigned long long)want), 1;
            }
        }
    return 0;
}
"""


def test_walk_ends_and_takes_every_item(tmp_path):
    src, exe = tmp_path / "walk.cu", tmp_path / "walk"
    src.write_text(PROGRAM)
    subprocess.run([build.nvcc(), "-std=c++17", "-O1", "-I", build.CSRC, "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_no_32_bit_index_steps_by_the_grid():
    """Loops over a grid's items use Strided or a 64-bit index."""
    loop = re.compile(r"for \(uint32_t (\w+) = blockIdx\.x \* blockDim\.x \+ threadIdx\.x;")
    for f in sorted(os.listdir(build.CSRC)):
        if f.endswith((".cu", ".cuh", ".h")):
            with open(os.path.join(build.CSRC, f)) as src:
                assert not loop.search(src.read()), f
