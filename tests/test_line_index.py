"""The line kernel's arithmetic that the host shares (line_index.cuh), with
signed overflow trapping: for every image it takes, the smallest and the
largest included, the corners' indices are those of 64-bit arithmetic; a quotient by
a multiplication is the division's, bit for bit; the blocks of the rows'
contraction are resident at once where the split says so, whatever the
device's number of SMs."""
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


QUOTIENT = r"""
#include <cstdint>
#include "line_index.cuh"
using namespace b200;

int main ()
{
    uint64_t r = 88172645463325252ull;
    auto uniform = [&] {
        r ^= r << 13; r ^= r >> 7; r ^= r << 17;
        return (float) (r >> 40) / 16777216.f;
    };
    // image ranges of 2^-20 to 2^30 grey levels, 5 to 64 bins
    for (int t = 0; t < 2000; t++) {
        const float range = std::exp2 (-20.f + 50.f * uniform ());
        const float d = range / (float) (1 + (int) (60.f * uniform ()));
        for (int k = 0; k < 1000; k++) {
            const float x = range * uniform ();
            volatile float want = x / d;
            if (line_quotient (x, d, 1.f / d) != want) return 1;
        }
    }
    return 0;
}
"""

SPLIT = r"""
#include <initializer_list>
#include "line_index.cuh"
using namespace b200;

int main ()
{
    const int sizes[] = {4, 7, 14, 23, 40, 55, 108, 160};
    int resident = 0, waves = 0;
    for (int sms : {20, 74, 132, 148, 160})
    for (int vx : {3, 5, 8, 10}) for (int vz : {3, 5, 8, 10})
    for (int cx : sizes) for (int cy : sizes) for (int cz : sizes) {
        const int c[3] = {cx, cy, cz}, v[3] = {vx, 5, vz};
        const LineSplit f = line_finish_split (c, v, sms);
        const int block = f.threads * f.parts;
        if (f.kxc * f.nbx < cx || f.kzc < 1 || f.kzc > 8 || f.parts > vz) return 1;
        if (2 * f.threads < (f.kxc + 3) * vx + 1 || f.threads % 32) return 2;
        if (block > LINE_SPLIT_THREADS) return 3;
        const int n = f.nbx * cy * ((cz + f.kzc - 1) / f.kzc);
        if (!f.waves && n > sms * (LINE_SPLIT_THREADS / block)) return 4;
        (f.waves ? waves : resident)++;
    }
    return resident > 1000 && waves > 1000 ? 0 : 5;
}
"""


def _build(tmp_path_factory, name, text):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp(name)
    src, exe = d / "main.cpp", d / "main"
    src.write_text(text)
    subprocess.run([cxx, "-std=c++17", "-O1", "-ffp-contract=off",
                    "-fsanitize=undefined",
                    "-fsanitize-undefined-trap-on-error", "-x", "c++", "-I",
                    os.path.join(ROOT, "plastimatch_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    return str(exe)


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return _build(tmp_path_factory, "index", PROGRAM)


@pytest.mark.parametrize("dim", [(2, 2, 2), (3, 2, 5), (64, 64, 64),
                                 (131, 117, 83), (512, 512, 160),
                                 (1023, 1025, 1024), (1 << 22, 2, 127)])
def test_corner_index(program, dim):
    assert subprocess.run([program] + [str(v) for v in dim]).returncode == 0


def test_quotient(tmp_path_factory):
    exe = _build(tmp_path_factory, "quotient", QUOTIENT)
    assert subprocess.run([exe]).returncode == 0


def test_contraction_split(tmp_path_factory):
    exe = _build(tmp_path_factory, "split", SPLIT)
    assert subprocess.run([exe]).returncode == 0
