"""The edges of the kernels' dispatch: sizes, batches, layouts and alignments
on both sides of each rule, compared bit by bit with the oracle or with another
path to the same result."""
import numpy as np
import pytest

import oracle as O
import pcrp
from helpers import assert_bitexact, dd_bands, gpu_f64, to_device, to_layout, zero_bands

pytestmark = pytest.mark.gpu


def mixed(arrs, m, n, layout=pcrp.CONTIGUOUS, shift=0, **kw):
    """x of a mixed solve; shift: the arrays start `shift` doubles past an aligned address."""
    import torch
    t = []
    for v in arrs:
        if v is None:
            t.append(None)
            continue
        buf = torch.empty(m * n + shift, dtype=torch.float64, device="cuda:0")[shift:]
        buf.copy_(torch.from_numpy(np.ascontiguousarray(v)))
        t.append(buf)
    kw.setdefault("report", False)
    info = pcrp.solve_mixed(*t, m, n, layout, **kw)
    torch.cuda.synchronize()
    return t[5].cpu().numpy(), info


# ---------------------------------------------------------------------------
# FP64
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("n", [31, 32, 97, 384, 385, 544, 2047, 2048, 2049])
@pytest.mark.parametrize("m", [1, 37, 420])
def test_one_case_and_per_case_rows_bitexact(cuda, n, m):
    """Few or many CTAs, systems up to and past the short ones: one row case
    for all rows, or a case per kind of row."""
    for arrs in (dd_bands(np.random.default_rng(n + m), m, n),
                 zero_bands(np.random.default_rng(n * m), m, n, special=True)):
        x, _ = gpu_f64(arrs, m, n)
        assert_bitexact(x, O.pcr(*arrs, m, n), f"n={n} m={m}")


def tridiagonal(kind, rng, m, n):
    arrs = dd_bands(rng, m, n)
    a, b, c, d, e, y = arrs
    a[:] = 0.0
    e[:] = 0.0
    if kind == "overflow":                        # right-hand sides that pass the largest double in some stride
        y *= 1.7e308
    elif kind == "zeros":                         # single zeros among the coefficients and right-hand sides
        for v in (b, d, y):
            v[rng.random(m * n) < 0.03] = 0.0
    elif kind == "late inf":                      # one infinite coefficient, far from most rows
        c.reshape(m, n)[0, n // 2] = np.inf
    return arrs


@pytest.mark.parametrize("n", [3, 64, 513, 3001])
@pytest.mark.parametrize("kind", ["dominant", "overflow", "zeros", "late inf"])
def test_tridiagonal_rows_without_their_neighbours_bitexact(cuda, n, kind):
    """Null outer bands: rows formed alone while a tile is finite, and as
    before once it holds an infinity or zeros; uniform and ragged batches."""
    import torch
    m = 3
    arrs = tridiagonal(kind, np.random.default_rng(n), m, n)
    ref = O.pcr(*arrs, m, n)
    t = to_device(arrs, "cuda:0")
    t[0] = t[4] = None
    r = t[5].clone()
    pcrp.solve_f64(*t, m, n)
    offsets = torch.arange(m + 1, dtype=torch.int64, device="cuda:0") * n
    pcrp.solve_ragged(*t[:5], r, offsets, m, n)
    torch.cuda.synchronize()
    assert_bitexact(t[5].cpu().numpy(), ref, f"{kind} n={n}")
    assert_bitexact(r.cpu().numpy(), ref, f"ragged {kind} n={n}")


# ---------------------------------------------------------------------------
# mixed precision
# ---------------------------------------------------------------------------

@pytest.mark.parametrize("n", [4097, 4098, 5374, 5376, 5377, 8960, 30001])
@pytest.mark.parametrize("drop", [(), (0, 4), (4,)])
def test_inner_windows_match_the_general_form(cuda, n, drop):
    """Aligned windows inside a system address one run of rows; arrays that
    start 8 bytes past an aligned address take the general form everywhere.
    Window edges (1792 rows apart), odd sizes (every other system unaligned)."""
    m = 3
    arrs = dd_bands(np.random.default_rng(n), m, n, garbage=True)
    for k in drop:
        arrs[k] = None
    x, _ = mixed(arrs, m, n)
    xg, _ = mixed(arrs, m, n, shift=1)
    assert_bitexact(x, xg, f"n={n} null {drop}")


@pytest.mark.parametrize("n", [4099, 9000])
def test_coupled_systems_leave_the_others_alone(cuda, n):
    """Systems whose windows stay coupled send the solve through the general
    passes; the others of the batch keep the bits of a solve without them."""
    easy = dd_bands(np.random.default_rng(n), 2, n)
    hard = [np.asarray(v) for v in pcrp.generate(pcrp.GEN_ADI, 4, 2, n)]
    for _ in range(3):                            # first calls, then from a graph
        alone, _ = mixed(easy, 2, n, max_sweeps=16)
        both, _ = mixed([np.concatenate(v) for v in zip(easy, hard)], 4, n, max_sweeps=16)
        assert_bitexact(both[:2 * n], alone, f"n={n}")
    assert O.fwd_err(both[2 * n:], O.ge(*hard, 2, n), 2, n) <= 1e-12


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 63, 64, 65, 127, 128, 129, 255, 257, 510, 513, 1025, 2046, 2049, 4095, 4096])
def test_whole_systems_zero_and_null_outer_bands(cuda, n):
    """Whole systems (every sweep after the first replays the reduction on its
    rhs): an outer band of zeros gives the bits of a null one, also beside
    systems where it is not zero, and every system those of a solve alone."""
    arrs = dd_bands(np.random.default_rng(n), 3, n, garbage=True)
    rows = [v.reshape(3, n) for v in arrs]
    rows[0][0, 2:] = 0.0                          # (slots outside the system hold garbage)
    rows[4][2, :max(n - 2, 0)] = 0.0
    x, _ = mixed(arrs, 3, n, max_sweeps=5, tol=1e-16)
    for j in range(3):
        one = [v[j].copy() for v in rows]
        if j == 0:
            one[0] = None
        if j == 2:
            one[4] = None
        xj, _ = mixed(one, 1, n, max_sweeps=5, tol=1e-16)
        assert_bitexact(x[j * n:(j + 1) * n], xj, f"n={n} system {j}")
    xg = O.ge(*arrs, 3, n)
    assert O.fwd_err(x, xg, 3, n) <= 1e-12


@pytest.mark.parametrize("n", [2, 3, 1023, 1025, 4097, 9001])
@pytest.mark.parametrize("layout", [pcrp.CONTIGUOUS, pcrp.INTERLEAVED])
@pytest.mark.parametrize("drop", [(), (0, 4)])
def test_report_values(cuda, n, layout, drop):
    """The one-pass report: x as without a report, and the residual ratio of
    the separate residual (the maxima are rounded to single precision, 2^-24
    each, and the largest row sum is found from single-precision estimates)."""
    import torch
    m = 5
    arrs = dd_bands(np.random.default_rng(n), m, n)
    for k in drop:
        arrs[k][:] = 0.0
    lay = to_layout(arrs, m, n, layout)
    given = [None if k in drop else v for k, v in enumerate(lay)]
    for _ in range(2):                            # a first call, then from a graph
        x, info = mixed(given, m, n, layout, report=True)
        assert_bitexact(x, mixed(given, m, n, layout)[0], f"n={n}")
        t = to_device(lay + [x], "cuda:0")
        r = torch.empty_like(t[6])
        pcrp.residual_f64(*t, r, m, n, layout)
        back = (lambda v: v.reshape(m, n)) if layout == pcrp.CONTIGUOUS else (lambda v: v.reshape(n, m).T)
        top = [np.abs(back(v)).max(axis=1) for v in (r.cpu().numpy(), x)]
        rowsum = sum(np.abs(v.reshape(m, n)) for v in arrs[:5]).max(axis=1)
        want = (top[0] / (rowsum * top[1])).max()
        assert abs(info.resid - want) <= 2.0 ** -22 * want
        assert info.converged == 1
