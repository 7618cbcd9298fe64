"""The FP64 tile's row cases in the kernels that take a case per kind of row.

Pentadiagonal batches of at most 2048 rows, and launches of at most two warps
per SM sub-partition, run one case for all rows; a case per kind of row runs in
longer systems of larger batches and in every ragged batch.  The batches here
are of those: m=128 systems of more than 2048 rows are at least 128 * 5 tiles
of 5 or more warps in every pass, against 1216 warps on a GB300.  Every kind of
operands is compared with the oracle bit by bit."""
import numpy as np
import pytest

import oracle as O
import pcrp
from helpers import assert_bitexact, dd_bands, gpu_f64, to_device
from test_ieee_int import bands

pytestmark = pytest.mark.gpu

KINDS = ["tiny", "a0", "e0", "holes", "dyadic", "huge", "rows", "a0 holes", "e0 holes", "uneven"]


def operands(kind, rng, m, n):
    if kind == "rows":                            # rows scaled far apart: in and outside the window side by side
        arrs = dd_bands(rng, m, n)
        s = np.ldexp(1.0, rng.integers(-400, 401, m * n))
        for v in arrs:
            v *= s
        return arrs
    if kind == "uneven":                          # half of each system with small couplings: they underflow earlier
        arrs = dd_bands(rng, m, n)
        for v in (arrs[0], arrs[1], arrs[3], arrs[4]):
            v.reshape(m, n)[:, n // 2:] *= 1e-7
        return arrs
    if kind.endswith(" holes"):
        arrs = bands("holes", rng, m, n)
        z = np.where(rng.random(m * n) < 0.5, 0.0, -0.0)
        arrs[0 if kind[0] == "a" else 4][:] = z
        return arrs
    return bands(kind, rng, m, n)


@pytest.mark.parametrize("n", [2049, 4096, 9001])
@pytest.mark.parametrize("kind", KINDS)
def test_cases_per_kind_of_row_bitexact(cuda, n, kind):
    m = 128
    arrs = operands(kind, np.random.default_rng(n), m, n)
    x, _ = gpu_f64(arrs, m, n)
    assert_bitexact(x, O.pcr(*arrs, m, n), f"{kind} n={n}")


@pytest.mark.parametrize("drop", [0, 4])
@pytest.mark.parametrize("kind", ["tiny", "holes", "rows"])
def test_one_null_band_per_kind_of_row_bitexact(cuda, kind, drop):
    """One outer band null: row_a_one and its mirror image in every row."""
    m, n = 128, 3001
    arrs = operands(kind, np.random.default_rng(drop), m, n)
    arrs[drop][:] = 0.0
    import torch
    t = to_device(arrs, "cuda:0")
    pcrp.solve_f64(*[None if k == drop else v for k, v in enumerate(t)], m, n)
    torch.cuda.synchronize()
    assert_bitexact(t[5].cpu().numpy(), O.pcr(*arrs, m, n), f"{kind} null {drop}")


@pytest.mark.parametrize("opts", [dict(smem_rows=5, fuse_strides=2), dict(smem_rows=33, fuse_strides=1, tile_rows=31),
                                  dict(smem_rows=64, fuse_strides=3, threads=32), dict(smem_rows=1024), dict(smem_rows=1920)])
@pytest.mark.parametrize("kind", ["dyadic", "holes", "rows"])
def test_cases_across_passes_bitexact(cuda, kind, opts):
    """Small tiles: exact zero pivots and the multipliers carried from one pass
    to the next in the kernels with a case per kind of row; large ones."""
    m, n = 128, 2500
    arrs = operands(kind, np.random.default_rng(7), m, n)
    x, _ = gpu_f64(arrs, m, n, opts=pcrp.Opts(**opts))
    assert_bitexact(x, O.pcr(*arrs, m, n), f"{kind} {opts}")


@pytest.mark.parametrize("kind", KINDS)
def test_ragged_cases_bitexact(cuda, kind):
    """Ragged batches take a case per kind of row at every size: systems of a
    warp, of a tile, of two and more passes."""
    import torch
    rng = np.random.default_rng(11)
    sizes = [1, 2, 3, 5, 31, 32, 33, 64, 200, 511, 512, 513, 700, 1024, 2047, 2049, 4096, 5000, 9001]
    parts = [operands(kind, rng, 1, n) for n in sizes]
    flat = [np.concatenate([q[k] for q in parts]) for k in range(6)]
    t = to_device(flat, "cuda:0")
    offsets = torch.from_numpy(np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)).to("cuda:0")
    pcrp.solve_ragged(*t, offsets, len(sizes), max(sizes))
    torch.cuda.synchronize()
    x = t[5].cpu().numpy()
    at = 0
    for n, q in zip(sizes, parts):
        assert_bitexact(x[at:at + n], O.pcr(*q, 1, n), f"{kind} n={n}")
        at += n


@pytest.mark.parametrize("n", [3, 33, 64, 513, 3001])
@pytest.mark.parametrize("spread", [400, 900])
def test_tridiagonal_rows_scaled_apart_bitexact(cuda, n, spread):
    """Null outer bands and rows scaled by up to 2^+-400 (quotients inside the
    integer quotient's guard, products outside the integer product's window)
    and 2^+-900 (quotients outside it as well, subnormal and overflowing
    ones); uniform and ragged."""
    import torch
    m = 5
    rng = np.random.default_rng(n + spread)
    arrs = dd_bands(rng, m, n)
    s = np.ldexp(1.0, rng.integers(-spread, spread + 1, m * n))
    for v in arrs:
        v *= s
    arrs[0][:] = 0.0
    arrs[4][:] = 0.0
    for v in (arrs[1], arrs[3]):                  # signed zeros among the couplings
        v[rng.random(m * n) < 0.05] = -0.0
    ref = O.pcr(*arrs, m, n)
    t = to_device(arrs, "cuda:0")
    t[0] = t[4] = None
    r = t[5].clone()
    pcrp.solve_f64(*t, m, n)
    offsets = torch.arange(m + 1, dtype=torch.int64, device="cuda:0") * n
    pcrp.solve_ragged(*t[:5], r, offsets, m, n)
    torch.cuda.synchronize()
    assert_bitexact(t[5].cpu().numpy(), ref, f"n={n} spread={spread}")
    assert_bitexact(r.cpu().numpy(), ref, f"ragged n={n} spread={spread}")


@pytest.mark.parametrize("opts", [None, dict(smem_rows=5, fuse_strides=2), dict(smem_rows=33, fuse_strides=1, tile_rows=31),
                                  dict(smem_rows=64, fuse_strides=3, threads=32)])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 33, 64, 90, 513, 3001])
@pytest.mark.parametrize("kind", ["dyadic", "holes", "spike"])
def test_tridiagonal_zeros_and_zero_pivots_bitexact(cuda, kind, n, opts):
    """Null outer bands with zeros of both signs anywhere: exact zero pivots,
    also in the last stride and across passes, and zero right-hand sides but
    for one value per system; uniform and ragged."""
    import torch
    m = 40
    rng = np.random.default_rng(n)
    arrs = operands("holes" if kind == "spike" else kind, rng, m, n)
    if kind == "spike":
        arrs[5][:] = 0.0
        arrs[5].reshape(m, n)[:, n // 2] = 1.0
    arrs[0][:] = 0.0
    arrs[4][:] = 0.0
    for v in (arrs[1], arrs[2], arrs[3], arrs[5]):
        z = (v == 0.0) & (rng.random(m * n) < 0.5)
        v[z] = -0.0
    ref = O.pcr(*arrs, m, n)
    t = to_device(arrs, "cuda:0")
    t[0] = t[4] = None
    r = t[5].clone()
    o = pcrp.Opts(**opts) if opts else None
    pcrp.solve_f64(*t, m, n, opts=o)
    assert_bitexact(t[5].cpu().numpy(), ref, f"{kind} n={n} {opts}")
    if not opts:
        offsets = torch.arange(m + 1, dtype=torch.int64, device="cuda:0") * n
        pcrp.solve_ragged(*t[:5], r, offsets, m, n)
        assert_bitexact(r.cpu().numpy(), ref, f"ragged {kind} n={n}")
