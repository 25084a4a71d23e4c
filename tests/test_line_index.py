"""The line kernel's corner index (line_index.cuh) on the host, with signed
overflow trapping: for every image it takes, the smallest and the largest
included, the corners' indices are those of 64-bit arithmetic."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include "line_index.cuh"
using namespace b200;

static int bits_of (int i)
{
    const float f = 8388608.f + (float) i;
    int b;
    memcpy (&b, &f, 4);
    return b;
}

int main (int argc, char** argv)
{
    int n[3];
    if (argc != 4) return 2;
    for (int d = 0; d < 3; d++) sscanf (argv[1 + d], "%d", n + d);
    const unsigned c0 = line_corner0 (n[0], n[1]);
    for (int k = 0; k < 125; k++) {
        int i[3], b[3];
        for (int d = 0, r = k; d < 3; d++, r /= 5) {
            const int at[5] = {0, 1, n[d] / 2, n[d] - 2, n[d] - 1};
            i[d] = at[r % 5];
            b[d] = bits_of (i[d]);
        }
        const long long want = i[0] + (long long) n[0] * (i[1] + (long long) n[1] * i[2]);
        if ((long long) line_corner (b, n[0], n[1], c0) != want) return 1;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("line_index")
    src, exe = d / "index.cpp", d / "index"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-fsanitize=undefined",
                    "-fsanitize-undefined-trap-on-error", "-x", "c++", "-I",
                    os.path.join(ROOT, "plastimatch_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("dim", [(2, 2, 2), (3, 2, 5), (64, 64, 64),
                                 (131, 117, 83), (512, 512, 160),
                                 (1023, 1025, 1024), (1 << 22, 2, 127)])
def test_corner_index(program, dim):
    assert subprocess.run([program] + [str(v) for v in dim]).returncode == 0
