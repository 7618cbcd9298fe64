"""Products and quotients formed on the integer pipe (csrc/ieee_int.cuh) and
the FP64 tile's row cases built on them: bit equality with IEEE arithmetic and
with the oracle."""
import os
import subprocess

import numpy as np
import pytest

import oracle as O
import pcrp
from helpers import assert_bitexact, dd_bands, gpu_f64

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pcr-penta_gb300", "csrc")

HOST = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "ieee_int.cuh"
using namespace pcrp;
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s * 0x2545F4914F6CDD1Dull; }
static double gen(int mode) {                       // mantissas: random, near all ones or 1, one bit, trailing zeros
    uint64_t m = rnd() >> 12, r = rnd(), e = (r >> 20) % 2048;
    if (mode & 4) e = 1023 + (r >> 20) % 64 - 32;
    if ((mode & 3) == 1) m = (r & 1) ? 0xFFFFFFFFFFFFFull - rnd() % 16 : rnd() % 16;
    if ((mode & 3) == 2) { m = 1ull << (r % 52); if (r & 64) m -= rnd() % 4; m &= 0xFFFFFFFFFFFFFull; }
    if ((mode & 3) == 3) m &= ~((1ull << (r % 52)) - 1);
    const uint64_t u = (rnd() & (1ull << 63)) | (e << 52) | m;
    double d; memcpy(&d, &u, 8); return d;
}
int main() {
    long bad = 0, n[3] = {0, 0, 0};
    for (int i = 0; i < 4000000; i++) {
        const int mo = rnd() % 64;
        const double x = gen(mo & 7), y = gen(mo >> 3);
        const volatile double p = x * y, q = x / y;
        double r;
        if (ieee::mid(x) && ieee::mid(y)) { r = ieee::mul(ieee::factor(x), y); bad += memcmp((void*)&p, &r, 8) != 0; n[0]++; }
        if (ieee::div_guard(x, y)) { r = ieee::div(x, y, ieee::recip(y)); bad += memcmp((void*)&q, &r, 8) != 0; n[1]++; }
        if (ieee::div_any(x, y, r)) { bad += memcmp((void*)&q, &r, 8) != 0; n[2]++; }
    }
    printf("%ld %ld %ld %ld\n", bad, n[0], n[1], n[2]);
}
"""


def test_integer_products_and_quotients_are_ieee(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(HOST)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    bad, nm, nd, na = map(int, subprocess.run([str(tmp_path / "t")], check=True, capture_output=True,
                                              text=True).stdout.split())
    assert bad == 0
    assert min(nm, nd, na) > 500000               # every function saw its share of operands


def bands(kind, rng, m, n):
    arrs = dd_bands(rng, m, n)
    a, b, c, d, e, y = arrs
    if kind == "tiny":                            # couplings that run through the subnormals at different strides
        for v in (a, b, d, e):
            v *= 10.0 ** rng.uniform(-60, 0, m * n)
    elif kind == "a0":
        a[:] = 0.0
    elif kind == "e0":
        e[:] = np.where(rng.random(m * n) < 0.5, 0.0, -0.0)
    elif kind == "holes":                         # single zeros among the outer and inner coefficients and the rhs
        for v in (a, b, d, e, y):
            v[rng.random(m * n) < 0.02] = 0.0
    elif kind == "dyadic":                        # small integers: pivots that cancel to zero exactly
        for v in arrs:
            v[:] = rng.integers(-2, 3, m * n)
    elif kind == "huge":                          # outside the window of the integer row cases
        for v in arrs:
            v *= 2.0 ** rng.integers(-450, 450)
    return arrs


@pytest.mark.gpu
# one row case short of / at / past: the short-system limit (320), the tile (512), its window with halos (544), two
# and more passes; odd, and powers of two
# (The short-system limit is 2048 rows since, so these batches run the one case for all rows; test_row_cases_gpu.py
# runs the same kinds in the kernels that take a case per kind of row.)
@pytest.mark.parametrize("n", [3, 33, 320, 321, 512, 513, 1023, 1024, 1090, 4096, 9001])
@pytest.mark.parametrize("kind", ["tiny", "a0", "e0", "holes", "dyadic", "huge"])
def test_row_cases_bitexact(cuda, n, kind):
    rng = np.random.default_rng(n)
    for m in (3, 700) if n <= 1090 else (3,):     # few CTAs (general rows) and a full machine
        arrs = bands(kind, rng, m, n)
        x, _ = gpu_f64(arrs, m, n)
        assert_bitexact(x, O.pcr(*arrs, m, n), f"{kind} n={n} m={m}")


@pytest.mark.gpu
@pytest.mark.parametrize("opts", [dict(smem_rows=2), dict(smem_rows=3, fuse_strides=1), dict(smem_rows=5, fuse_strides=2)])
def test_last_strides_across_passes_bitexact(cuda, opts):
    """Tiles of a few rows: the last strides, whose zero pivots reuse a kept
    multiplier, fall into different passes."""
    for n in (7, 12, 33, 64, 100):
        rng = np.random.default_rng(n)
        arrs = bands("dyadic", rng, 40, n)
        x, _ = gpu_f64(arrs, 40, n, opts=pcrp.Opts(**opts))
        assert_bitexact(x, O.pcr(*arrs, 40, n), f"n={n} {opts}")


COMPOSED = HOST.split("static double gen")[0] + r"""
static double make(int e, uint64_t m) {
    const uint64_t u = (rnd() & (1ull << 63)) | ((uint64_t)e << 52) | (m & 0xFFFFFFFFFFFFFull);
    double d; memcpy(&d, &u, 8); return d;
}
static double end() {                               // the window's ends, mantissas near all ones or a power of two
    const uint64_t r = rnd(), m = (r & 4) ? ~(rnd() % 16) : rnd() % 16;
    return make((r & 1) ? 623 + (r >> 8) % 2 : 1134 - (r >> 8) % 2, (r & 8) ? m : rnd() >> 12);
}
static double odd(int bits) {                       // an odd integer of so many bits, scaled into [1, 2)
    const uint64_t unit = 1ull << (53 - bits);
    return make(1015 + rnd() % 16, bits == 1 ? 0 : ((rnd() >> 12) & ~(2 * unit - 1)) | unit);
}
static bool same(double x, const volatile double& y) { return memcmp(&x, (const void*)&y, 8) == 0; }
int main() {
    long bad = 0, outside = 0, ties = 0;
    for (int i = 0; i < 4000000; i++) {
        const double x = end(), y = end(), z = end();
        const volatile double q = x / y, p = q * z;
        const double g = ieee::div(x, y, ieee::recip(y));
        bad += !same(g, q) || !same(ieee::mul(ieee::factor(g), z), p);
        outside += !ieee::mid(g);
        const int k = 2 + rnd() % 51;
        const double a = odd(k), b = odd(54 - k + rnd() % 2);
        const volatile double r = a * b;
        bad += !same(ieee::mul(ieee::factor(a), b), r);
        ties += __builtin_fma(a, b, -r) != 0.0;
    }
    printf("%ld %ld %ld\n", bad, outside, ties);
}
"""


def test_products_of_quotients_and_ties_are_ieee(tmp_path):
    """Products as the kernels form them: a quotient of two window operands,
    whose exponent may lie outside `mid`, times a third; and products half way
    between two doubles."""
    src = tmp_path / "t.cpp"
    src.write_text(COMPOSED)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(tmp_path / "t")], check=True)
    bad, outside, ties = map(int, subprocess.run([str(tmp_path / "t")], check=True, capture_output=True,
                                                 text=True).stdout.split())
    assert bad == 0
    assert outside > 100000 and ties > 1000000


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4])
def test_integer_arithmetic_on_the_device_is_ieee(cuda, mode):
    """The device code (its own carry chains) one operation at a time."""
    samples = 1 << 27
    bad, products, quotients, any_size = pcrp.check_integer_arithmetic(mode, 77 + mode, samples)
    assert bad == 0
    # shares: every triple but in mode 4, where exponents of the window are (512/2048)^3 of them and sums that
    # leave the product normal about 3/4
    assert products >= (samples // 2 if mode == 4 else samples)
    assert quotients >= (samples // 128 if mode == 4 else samples)
    assert any_size >= samples // 4


def test_integer_arithmetic_check_refuses_bad_arguments(built_lib):
    import ctypes
    counts = (ctypes.c_uint64 * 4)()
    f = pcrp.lib().pcrp_check_integer_arithmetic
    assert f(-1, 0, 1, counts, None) == 1
    assert f(5, 0, 1, counts, None) == 1
    assert f(0, 0, -1, counts, None) == 1
    assert f(0, 0, 1, None, None) == 1
