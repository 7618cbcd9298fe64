"""Performance cases of the batched pentadiagonal solvers.

A case is a plain dict; `prepare` makes what a program holds before the call
(bands and right-hand side, on the device or in host memory), `run` is one
call through the public Python entry points, `work` the bytes and operations
one call cannot do without and `exact` its result in 64 bits from plain torch.

Entries (`entry`):
  f64     pcrp.solve_f64, the FP64 PCR solve in place on a copy of the rhs
  mixed   pcrp.solve_mixed, FP32 reduction + FP64 refinement (with or without
          the per-call report)
  step    one theta step of the ADI driver: rhs = B u (pcrp.residual_f64 on
          the negated explicit operator), copy, mixed solve
  ragged  pcrp.solve_ragged on systems of uneven size, mode 0 FP64, 1 mixed
  host    pcrp.solve_host on page-locked host arrays, waiting for the result
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "pcr-penta_gb300"))

import pcrp  # noqa: E402

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # the smallest call: a handful of short systems of no special size inside a larger program (latency, launches)
        dict(name="f64_few_short", entry="f64", m=8, n=100, kind="dominant", layout="contiguous", tri=False),
        # many short systems, interleaved batch format: one line solve of a 2D grid
        dict(name="f64_short_interleaved", entry="f64", m=1024, n=512, kind="dominant", layout="interleaved", tri=False),
        # tridiagonal batch (null outer bands), size not a power of two
        dict(name="f64_tridiagonal_odd", entry="f64", m=777, n=3001, kind="dominant", layout="contiguous", tri=True),
        # long systems, the size the method's published tables end at
        dict(name="f64_long", entry="f64", m=256, n=65536, kind="dominant", layout="contiguous", tri=False),
        # the benchmark's own workload: few very long, weakly dominant systems
        dict(name="f64_longest", entry="f64", m=64, n=1 << 20, kind="weak", layout="contiguous", tri=False),
        # uneven systems, FP64, log-uniform sizes
        dict(name="ragged_f64", entry="ragged", nsys=4096, nmin=32, nmax=65536, kind="dominant", mode=0),
        # many short systems in mixed precision, interleaved
        dict(name="mixed_short_interleaved", entry="mixed", m=1024, n=512, kind="dominant", layout="interleaved", tri=False, report=False),
        # mixed precision with the per-call report (the Python default), odd size
        dict(name="mixed_report_odd", entry="mixed", m=100, n=30001, kind="dominant", layout="contiguous", tri=False, report=True),
        # few very long, weakly dominant systems in mixed precision
        dict(name="mixed_longest", entry="mixed", m=64, n=1 << 20, kind="weak", layout="contiguous", tri=False, report=False),
        # one time step of the batched option-pricing driver
        dict(name="adi_step", entry="step", m=4096, n=4096),
        # uneven systems, mixed precision
        dict(name="ragged_mixed", entry="ragged", nsys=4096, nmin=32, nmax=65536, kind="dominant", mode=1),
        # a batch that lives in host memory, copies in and out included
        dict(name="host_mixed", entry="host", m=128, n=32768, kind="dominant", precision=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(["f64", "f64", "f64", "mixed", "mixed", "ragged", "step", "host"])
    if entry == "ragged":
        nmin = _log_int(rng, 16, 512)
        return dict(entry=entry, nsys=_log_int(rng, 64, 4096), nmin=nmin, nmax=_log_int(rng, 4 * nmin, 65536),
                    kind=rng.choice(["dominant", "weak"]), mode=rng.randrange(2))
    if entry == "step":
        n = _log_int(rng, 64, 8192)
        return dict(entry=entry, m=max(4, _log_int(rng, 1 << 14, 1 << 24) // n), n=n)
    # system sizes over the whole range, batches from a few thousand unknowns up
    n = _log_int(rng, 32, 1 << 20)
    if entry == "host":
        n = min(n, 1 << 18)
    total = _log_int(rng, max(n, 1 << 12), 1 << 22 if entry == "host" else 1 << 24)
    m = max(1, total // n)
    kind = rng.choice(["dominant", "weak", "adi"] if n <= 8192 else ["dominant", "weak"])
    if entry == "host":
        return dict(entry=entry, m=m, n=n, kind=kind, precision=rng.randrange(2))
    case = dict(entry=entry, m=m, n=n, kind=kind, layout=rng.choice(["contiguous", "contiguous", "interleaved"]),
                tri=rng.random() < 0.25)
    if entry == "mixed":
        case["report"] = rng.random() < 0.4
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _sizes(case):
    """Rows of each system of a ragged case: log-uniform, the same for every seed."""
    u = np.random.RandomState(97).random_sample(case["nsys"])
    lo, hi = case["nmin"], case["nmax"]
    return np.clip(np.round(lo * (hi / lo) ** u).astype(np.int64), lo, hi)


def _positions(case):
    """(row within its system, rows of that system) of every unknown, system after system."""
    if case["entry"] == "ragged":
        sizes = torch.from_numpy(_sizes(case)).to(DEVICE)
        n = torch.repeat_interleave(sizes, sizes)
        first = torch.repeat_interleave(torch.cumsum(sizes, 0) - sizes, sizes)
        return torch.arange(n.numel(), device=DEVICE) - first, n
    m, n = case["m"], case["n"]
    i = torch.arange(n, device=DEVICE).expand(m, n).reshape(-1)
    return i, n


def _adi_operator(case, g, i, coef):
    """Bands of I + coef*L of a convection-diffusion operator on S in [0, 800],
    second-order one-sided convection; `g` draws a variance per system."""
    m, n = case["m"], case["n"]
    v = torch.rand(m, generator=g, device=DEVICE, dtype=torch.float64) * 0.99 + 0.01
    h, r = 800.0 / (n - 1), 0.03
    S = torch.arange(n, device=DEVICE, dtype=torch.float64) * h
    diff = (0.5 * v[:, None] * (S * S)[None, :] / (h * h)).reshape(-1)
    conv = (r * S / (2.0 * h)).expand(m, n).reshape(-1)
    return [torch.zeros_like(diff), coef * diff, 1.0 + coef * (-2.0 * diff - 3.0 * conv - r),
            coef * (diff + 4.0 * conv), -coef * conv]


def _clip(bands, i, n):
    """Zeros in the slots that lie outside their system."""
    a, b, _, d, e = bands
    a.masked_fill_(i < 2, 0.0)
    b.masked_fill_(i < 1, 0.0)
    d.masked_fill_(i + 1 >= n, 0.0)
    e.masked_fill_(i + 2 >= n, 0.0)
    return bands


def _system(case, seed):
    """(bands, rhs) in the contiguous order, on the device, from the seed alone."""
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    i, n = _positions(case)

    def uniform(lo, hi):
        return torch.rand(i.numel(), generator=g, device=DEVICE, dtype=torch.float64) * (hi - lo) + lo

    kind = case.get("kind", "adi")
    if kind == "adi":
        bands = _clip(_adi_operator(case, g, i, -0.5e-3), i, n)
        strike = 50.0 + 100.0 * torch.rand(case["m"], generator=g, device=DEVICE, dtype=torch.float64)
        S = torch.arange(n, device=DEVICE, dtype=torch.float64) * (800.0 / (n - 1))
        y = torch.clamp(S[None, :] - strike[:, None], min=0.0).reshape(-1)
    else:
        a, b, d, e = [uniform(-1.0, 1.0) for _ in range(4)]
        _clip([a, b, None, d, e], i, n)
        if case.get("tri"):
            a.zero_()
            e.zero_()
        off = a.abs() + b.abs() + d.abs() + e.abs()
        if kind == "dominant":
            c = off + uniform(1.0, 2.0)
        else:
            c = torch.where(uniform(0.0, 1.0) < 0.5, -1.05, 1.05) * torch.clamp(off, min=1e-3)
        bands = [a, b, c, d, e]
        y = uniform(-1.0, 1.0)
    if case.get("tri"):
        bands[0].zero_()
        bands[4].zero_()
    return bands, y


def _to_layout(case, t):
    if case.get("layout") == "interleaved":
        return t.view(case["m"], case["n"]).t().contiguous().reshape(-1)
    return t


def prepare(case, seed):
    entry = case["entry"]
    bands, y = _system(case, seed)
    if case.get("tri"):
        bands[0] = bands[4] = None
    bands = [None if t is None else _to_layout(case, t) for t in bands]
    y = _to_layout(case, y)
    s = dict(case=case, bands=bands, rhs=y, x=torch.empty_like(y),
             layout=pcrp.INTERLEAVED if case.get("layout") == "interleaved" else pcrp.CONTIGUOUS)
    if entry == "step":
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed)                      # the same variances as the implicit operator
        i, n = _positions(case)
        s["explicit"] = [-t for t in _clip(_adi_operator(case, g, i, 0.5e-3), i, n)]
        s["zero"] = torch.zeros_like(y)
        s["out"] = torch.empty_like(y)
    elif entry == "ragged":
        off = np.concatenate([[0], np.cumsum(_sizes(case))])
        s["offsets"] = torch.from_numpy(off).to(DEVICE)
    elif entry == "host":
        host = []
        for t in bands + [y, y]:
            h = torch.empty(t.numel(), dtype=torch.float64, pin_memory=DEVICE == "cuda")
            h.copy_(t)
            host.append(h)
        s = dict(case=case, host=host[:5], rhs=host[5], x=host[6])
    return s


def run(s):
    case = s["case"]
    entry = case["entry"]
    x = s["x"]
    if entry == "step":
        m, n = case["m"], case["n"]
        pcrp.residual_f64(*s["explicit"], s["zero"], s["rhs"], s["out"], m, n)
        x.copy_(s["out"])
        pcrp.solve_mixed(*s["bands"], x, m, n, report=False)
        return [s["out"], x]
    x.copy_(s["rhs"])                            # the solvers overwrite the rhs
    if entry == "host":
        pcrp.solve_host(*s["host"], x, case["m"], case["n"], precision=case["precision"])
        torch.cuda.current_stream().synchronize()    # the result is read on the host
    elif entry == "ragged":
        pcrp.solve_ragged(*s["bands"], x, s["offsets"], case["nsys"], case["nmax"], mode=case["mode"])
    elif entry == "mixed":
        pcrp.solve_mixed(*s["bands"], x, case["m"], case["n"], s["layout"], report=case["report"])
    else:
        pcrp.solve_f64(*s["bands"], x, case["m"], case["n"], s["layout"])
    return x


# ---------------------------------------------------------------------------
# work and exact results
# ---------------------------------------------------------------------------

def _strides(n):
    """PCR strides of a system of n rows."""
    if n <= 1:
        return 0
    lg = (n - 1).bit_length()
    return lg if (1 << lg) == n else lg - 1


def work(case):
    if case["entry"] == "ragged":
        sizes = [int(v) for v in _sizes(case)]
    else:
        sizes = [case["n"]] * case["m"]
    rows = float(sum(sizes))
    bands = 3 if case.get("tri") else 5
    # the rhs is restored by a copy before the in-place solve
    nbytes = rows * 8.0 * (bands + 2 + 2)
    f64 = case["entry"] == "f64" or case.get("mode") == 0 or case.get("precision") == 0
    if f64:
        # 36 products and sums and 4 quotients per row and stride (half of it without outer bands)
        per = 20.0 if case.get("tri") else 40.0
        flops = sum(n * (per * _strides(n) + 1.0) for n in sizes) if case["entry"] == "ragged" else \
            rows * (per * _strides(case["n"]) + 1.0)
    else:
        # block elimination once, then per refinement a residual and a solve
        flops = rows * (60.0 if case.get("tri") else 100.0)
    if case["entry"] == "step":
        nbytes += rows * 8.0 * 7
        flops += rows * 10.0
    if case["entry"] == "host":
        nbytes -= rows * 16.0
    return {"bytes": nbytes, "flops": flops}


def _mm(A, B):
    return (A[:, :, None] * B[None]).sum(1)


def _mv(A, y):
    return (A * y[None]).sum(1)


def _inv(D):
    det = D[0, 0] * D[1, 1] - D[0, 1] * D[1, 0]
    return torch.stack([torch.stack([D[1, 1], -D[0, 1]]), torch.stack([-D[1, 0], D[0, 0]])]) / det


def _shift(A):
    """A of the previous index (zero before the first)."""
    return torch.cat([torch.zeros_like(A[..., :1]), A[..., :-1]], -1)


def _cyclic(L, D, U, Y):
    """Block tridiagonal systems of 2x2 blocks, arrays (2, 2, N) and (2, N), by block cyclic reduction."""
    N = Y.shape[-1]
    if N == 1:
        return _mv(_inv(D), Y)
    if N % 2:
        pad = [torch.zeros_like(t[..., :1]) for t in (L, D, U, Y)]
        pad[1][0, 0] = pad[1][1, 1] = 1.0
        return _cyclic(*[torch.cat([t, p], -1) for t, p in zip((L, D, U, Y), pad)])[..., :N]
    Le, De, Ue, Ye = [t[..., 0::2].contiguous() for t in (L, D, U, Y)]
    Lo, Do, Uo, Yo = [t[..., 1::2].contiguous() for t in (L, D, U, Y)]
    Di = _inv(Do)
    Lo, Uo, Yo = _mm(Di, Lo), _mm(Di, Uo), _mv(Di, Yo)       # odd rows with unit diagonal blocks
    Lm, Um, Ym = _shift(Lo), _shift(Uo), _shift(Yo)
    xe = _cyclic(-_mm(Le, Lm), De - _mm(Le, Um) - _mm(Ue, Lo), -_mm(Ue, Uo), Ye - _mv(Le, Ym) - _mv(Ue, Yo))
    xn = torch.cat([xe[..., 1:], torch.zeros_like(xe[..., :1])], -1)
    xo = Yo - _mv(Lo, xe) - _mv(Uo, xn)
    return torch.stack([xe, xo], -1).reshape(2, N)


def _multiply(bands, x):
    a, b, c, d, e = bands
    z = torch.zeros(2, dtype=x.dtype, device=x.device)
    xp = torch.cat([z, x, z])
    N = x.numel()
    return a * xp[0:N] + b * xp[1:N + 1] + c * x + d * xp[3:N + 3] + e * xp[4:N + 4]


def _solve(bands, y):
    """All systems end to end as one (the slots between them are zero), refined twice."""
    N = y.numel()
    if N % 2:
        one = [torch.zeros(1, dtype=y.dtype, device=y.device) for _ in range(6)]
        one[2] += 1.0
        return _solve([torch.cat([t, o]) for t, o in zip(bands, one)], torch.cat([y, one[5]]))[:N]
    a, b, c, d, e = [t.view(-1, 2).t() for t in bands]
    z = torch.zeros_like(c[0])
    L = torch.stack([torch.stack([a[0], b[0]]), torch.stack([z, a[1]])])
    D = torch.stack([torch.stack([c[0], d[0]]), torch.stack([b[1], c[1]])])
    U = torch.stack([torch.stack([e[0], z]), torch.stack([d[1], e[1]])])

    def once(r):
        return _cyclic(L, D, U, r.view(-1, 2).t()).t().reshape(-1)

    x = once(y)
    for _ in range(2):
        x = x + once(y - _multiply(bands, x))
    return x


def exact(case, seed):
    bands, y = _system(case, seed)
    if case["entry"] == "step":
        g = torch.Generator(device=DEVICE)
        g.manual_seed(seed)
        i, n = _positions(case)
        rhs = _multiply(_clip(_adi_operator(case, g, i, 0.5e-3), i, n), y)
        return [rhs, _solve(bands, rhs)]
    x = _to_layout(case, _solve(bands, y))
    return x.cpu() if case["entry"] == "host" else x
