"""Divisions done by a multiplication and one correction are the correctly rounded quotients.

Two of them carry the bit-exactness of the meshes: a coordinate by the weld quantum (k_mesh.cu,
quantum) and a sum of neighbours by their number (k_smooth.cu, gs_div).  The same operations in C, with
a fused multiply-add, against the division itself: every float where it matters.
"""
import ctypes
import subprocess

import pytest

SOURCE = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>

static float f(uint32_t b) { float x; memcpy(&x, &b, 4); return x; }

/* positions: floats of exponent e (biased), all mantissas; returns how many differ */
long long quantum(int e) {
    const volatile float one = 1.0f, tol = 0.001f;
    const float t = tol, r = one / t;
    long long bad = 0;
    for (uint32_t m = 0; m < 1u << 23; m++) {
        const float p = f((uint32_t)e << 23 | m), q = p * r;
        if (fmaf(fmaf(-q, t, p), r, q) != p / t) bad++;
    }
    return bad;
}

/* sums: all mantissas of one exponent, by a number of neighbours */
long long mean(int n, int e) {
    const volatile float one = 1.0f;
    const float d = (float)n, r = one / d;
    long long bad = 0;
    for (uint32_t m = 0; m < 1u << 23; m++) {
        const float s = f((uint32_t)e << 23 | m), q = s * r;
        if (fmaf(fmaf(-q, d, s), r, q) != s / d) bad++;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    (d / "division.c").write_text(SOURCE)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-o", str(d / "division.so"),
                    str(d / "division.c"), "-lm"], check=True)
    lib = ctypes.CDLL(str(d / "division.so"))
    for fn in (lib.quantum, lib.mean):
        fn.restype = ctypes.c_longlong
    return lib


def test_every_coordinate_by_the_quantum(lib):
    # 2^-13 (below, the quotient rounds to 0 either way) to the 16 384 that coordinates stay within
    assert sum(lib.quantum(e) for e in range(127 - 13, 127 + 14)) == 0


def test_every_sum_by_its_number_of_neighbours(lib):
    # an even number is an odd one times a power of two, and the exponent only scales; lists have up to 126
    assert sum(lib.mean(n, 127) for n in range(1, 127, 2)) == 0


@pytest.mark.parametrize("e", [127 - 100, 127 + 20, 254])  # the smallest sums taken so, and large ones
def test_the_exponent_only_scales(lib, e):
    assert sum(lib.mean(n, e) for n in (1, 2, 3, 6, 7, 100, 125, 126)) == 0
