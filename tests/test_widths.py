"""Places that a large call carries past the width of the integers they are made
from (csrc/widths.cuh).  The arithmetic is the kernels', run on the host; data
of that size is not."""
import os
import re
import subprocess

from test_host_tables import CSRC, cuda_include

PROGRAM = r"""
#include <stdio.h>
#include "widths.cuh"
int main() {
    const unsigned T = 256;
    const long long at[] = {0, 1, 7, 8, (1ll << 27) - 1, 1ll << 27, (1ll << 27) + 1, (1ll << 31) - 9};
    for (long long w : at)
        for (unsigned lane = 0; lane < 32; lane += 31) {
            const long long t = 32 * w + lane;
            if (rsg::warp_index((unsigned)(t / T), T, (unsigned)(t % T)) != w) {
                printf("warp %lld\n", w);
                return 1;
            }
        }
    printf("ok\n");
    return 0;
}
"""


POOL = r"""
#include <stdio.h>
#include "widths.cuh"
int main() {
    const int caps[] = {0, 1, 1000, 0x3fffffff};
    for (int cap : caps) {
        const unsigned long long at[] = {0, 1, 999, 1000, 0x3ffffffe, 0x3fffffff, 0x7fffffff,
                                         0x80000000u, 0x80000001u, 0xffffffffu};
        for (unsigned long long p : at)
            if (rsg::has_place((unsigned)p, cap) != (p < (unsigned long long)cap)) {
                printf("place %llu of %d\n", p, cap);
                return 1;
            }
    }
    printf("ok\n");
    return 0;
}
"""


def run(tmp_path, program):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(program)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", cuda_include(), str(src),
                           "-o", str(exe)])
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return f.read()


def test_beyond_two_to_the_27_warps(tmp_path):
    """The number of threads passes 2^32 there: the Barnes-Hut opening radii take
    a warp per tree node, and a call accepts records for more nodes than that."""
    run(tmp_path, PROGRAM)


def test_the_radii_use_it():
    s = source("props.cu")
    body = s[re.search(r"k_bh_dmin\(const KNode", s).end():][:600]
    assert "warp_index(blockIdx.x, blockDim.x, threadIdx.x)" in body


def test_list_chunks_beyond_two_to_the_31(tmp_path):
    run(tmp_path, POOL)


def test_the_lists_use_it():
    """The list builder asks it before it writes a chunk, and the number of
    chunks is the sum of the groups' in 64 bits, not the counter's last value."""
    s = source("fof3d.cu")
    assert "lost |= !has_place(nc, G.cap);" in s and "nc >= G.cap" not in s
    assert "cudaMemcpyAsync(&nch, go + ng" in s
