"""Batches that mix kinds of rows must not cost more than batches of the
costliest kind alone.

Every row of a batch scaled by 1e40 lies outside the integer row cases and
takes the FP64 path's general form.  A batch whose rows take different cases
(scattered zeros, exact zero pivots, rows scaled far apart) may run some of
them twice, but its warps then turn to the general form, so its time stays
near that of the scaled batch of the same size (bounds: what the extra tests
and the strides that try the cases again may cost; measured ratios beside
them).  Times are medians of CUDA-event timed solves."""
import numpy as np
import pytest

import oracle as O
import pcrp
from helpers import assert_bitexact, dd_bands, to_device

pytestmark = pytest.mark.gpu


def mix(kind, rng, m, n):
    arrs = dd_bands(rng, m, n)
    a, b, c, d, e, y = arrs
    if kind == "holes":
        for v in (a, b, d, e, y):
            v[rng.random(m * n) < 0.02] = 0.0
    elif kind == "dyadic":
        for v in arrs:
            v[:] = rng.integers(-2, 3, m * n)
    elif kind == "rows":
        s = np.ldexp(1.0, rng.integers(-400, 401, m * n))
        for v in arrs:
            v *= s
    elif kind == "scaled":
        for v in arrs:
            v *= 1e40
    return arrs


def solve_us(arrs, m, n, reps=15, null=()):
    """Median time of a solve (the bands in `null` not passed) and its solution."""
    import torch
    t = to_device(arrs, "cuda:0")
    rhs = t[5].clone()
    args = [None if k in null else v for k, v in enumerate(t)]
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(reps + 2):
        t[5].copy_(rhs)
        torch.cuda.synchronize()
        e0.record()
        pcrp.solve_f64(*args, m, n)
        e1.record()
        e1.synchronize()
        times.append(e0.elapsed_time(e1) * 1e3)
    return float(np.median(times[2:])), t[5].cpu().numpy()


# (with every row tried by the cases first: holes 1.9, dyadic 1.5-1.6, rows 1.7)
@pytest.mark.parametrize("kind", ["holes", "dyadic", "rows"])      # measured 1.05-1.07, 1.02-1.06, 1.3
@pytest.mark.parametrize("m,n", [(300, 2049), (256, 4096)])
def test_mixed_rows_cost_no_more_than_general_ones(cuda, kind, m, n):
    rng = np.random.default_rng(n)
    arrs = mix(kind, rng, m, n)
    us, x = solve_us(arrs, m, n)
    ref, _ = solve_us(mix("scaled", rng, m, n), m, n)
    print(f"\n[{kind} m={m} n={n}] {us:.1f} us, every row general {ref:.1f} us")
    assert_bitexact(x, O.pcr(*arrs, m, n), f"{kind} m={m} n={n}")
    assert us <= 1.45 * ref


# Short systems and few of them, where one case serves all rows: a warp's rows
# take it or the general form together (lane by lane: 1.4 and 1.5 times; now 1.0).
@pytest.mark.parametrize("m,n", [(8, 512), (4000, 128)])
def test_one_case_or_the_general_form(cuda, m, n):
    rng = np.random.default_rng(n)
    arrs = mix("rows", rng, m, n)
    us, x = solve_us(arrs, m, n)
    ref, _ = solve_us(mix("scaled", rng, m, n), m, n)
    print(f"\n[rows m={m} n={n}] {us:.1f} us, every row general {ref:.1f} us")
    assert_bitexact(x, O.pcr(*arrs, m, n), f"rows m={m} n={n}")
    assert us <= 1.25 * ref


# A tridiagonal batch (null outer bands) of widely scaled rows runs 10 of the
# pentadiagonal general form's 36 FP64 operations per row and stride and the
# same two quotients of phase B: with the general form it took 0.85 of the
# pentadiagonal batch's time, now 0.4.
@pytest.mark.parametrize("m,n", [(4000, 128)])
def test_tridiagonal_rows_outside_the_window(cuda, m, n):
    rng = np.random.default_rng(n)
    arrs = mix("rows", rng, m, n)
    ref, _ = solve_us(mix("scaled", rng, m, n), m, n)
    arrs[0][:] = 0.0
    arrs[4][:] = 0.0
    us, x = solve_us(arrs, m, n, null=(0, 4))
    print(f"\n[tridiagonal rows m={m} n={n}] {us:.1f} us, pentadiagonal, every row general {ref:.1f} us")
    assert_bitexact(x, O.pcr(*arrs, m, n), f"tridiagonal rows m={m} n={n}")
    assert us <= 0.7 * ref


# Tridiagonal batches of small integers decouple in a few strides while a tenth
# of their pivots are exactly zero.  Rows that divide by such a pivot took the
# pentadiagonal general form, and every row of a tile with one had the
# multipliers it leaves in place formed again: 0.95 to 1.35 of the time of a
# pentadiagonal batch whose rows all take the general form, now 0.58.
@pytest.mark.parametrize("m,n", [(4000, 128)])
def test_tridiagonal_rows_with_zero_pivots(cuda, m, n):
    rng = np.random.default_rng(n)
    arrs = mix("dyadic", rng, m, n)
    ref, _ = solve_us(mix("scaled", rng, m, n), m, n)
    arrs[0][:] = 0.0
    arrs[4][:] = 0.0
    us, x = solve_us(arrs, m, n, null=(0, 4))
    print(f"\n[tridiagonal zero pivots m={m} n={n}] {us:.1f} us, pentadiagonal, every row general {ref:.1f} us")
    assert_bitexact(x, O.pcr(*arrs, m, n), f"tridiagonal zero pivots m={m} n={n}")
    assert us <= 0.8 * ref
