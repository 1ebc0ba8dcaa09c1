"""How a plan cuts the tiles of contracted class pairs (csrc/bqc.h), on the CPU:
the ranges of the primitive quartets follow one another from the first to the
last, and the parts of a tile row fit the 32-bit row counts of the schedule."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r'''
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "bqc.h"
int main(int argc, char **argv) {
    for (int i = 1; i + 2 < argc; i += 3) {
        JKSub s;
        memset(&s, 0, sizeof(s));
        s.nprim_a = atoi(argv[i]);
        s.nprim_b = atoi(argv[i + 1]);
        s.na = s.nb = atoi(argv[i + 2]);
        split_prims(s);
        const long long n = (long long)s.nprim_a * s.nprim_b, cols = ((long long)s.nb + 15) / 16;
        bool ok = s.rparts >= 1 && s.rparts <= 8 && (s.rparts & (s.rparts - 1)) == 0 && s.kparts >= 1 &&
                  cols * s.rparts * s.kparts <= 0x7fffffffLL;
        long long at = 0;
        for (int k = 0; k < s.kparts && ok; k++) {
            const PrimRange r = prim_range(s, k);
            ok = r.num > 0 && r.k >= 0 && r.i >= 0 && r.i < s.nprim_a && (long long)r.k * s.nprim_a + r.i == at;
            at += r.num;
        }
        printf("%d", ok && at == n);
    }
    return 0;
}
'''

# primitive pairs of the bra and of the ket, pairs of each class: shells of 1, 3,
# 6, 24, 25 (25^4 / 64 * 25^4 is the first product above 2^31), 30 and 50 primitives,
# 216 (a quartet's number of primitives above 2^31), lists up to the 2^31 limit
CASES = [(a, b, n) for a, b in ((1, 1), (1, 36), (9, 9), (36, 36), (24 * 24, 24 * 24), (25 * 25, 25 * 25),
                                (1, 30 * 30), (30 * 30, 30 * 30), (50 * 50, 50 * 50), (216 * 216, 216 * 216))
         for n in (1, 17, 5000, 3000000, 2147483647)]


def test_primitive_ranges(tmp_path):
    nvcc = os.environ.get('NVCC', 'nvcc')
    if shutil.which(nvcc) is None:
        pytest.skip('nvcc not found')
    src, exe = tmp_path / 'ranges.cpp', tmp_path / 'ranges'
    src.write_text(SOURCE)
    subprocess.run([nvcc, '-std=c++17', '-O2', '-I', os.path.join(ROOT, 'byteqc_b200', 'csrc'),
                    '-I', os.path.join(ROOT, 'include'), str(src), '-o', str(exe)], check=True)
    out = subprocess.run([str(exe)] + [str(v) for c in CASES for v in c], check=True, capture_output=True,
                         text=True).stdout
    assert [c for c, ok in zip(CASES, out) if ok != '1'] == [] and len(out) == len(CASES)
