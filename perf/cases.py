"""Workloads of the SPME-RPY mobility operator, as its users run them, with the
inputs, one pass through the public entry points, the work that a pass cannot
do without, and the same result in 64 bits by plain torch.

Kinds of call (``"kind"`` of a case):

* ``step``: a time step on the device: new positions, then the operator on R
  right-hand sides (``Engine.set_positions`` + ``Engine.apply``, CUDA tensors);
* ``apply``: the operator at fixed positions, as one iteration of a block
  Lanczos / Krylov solver calls it, with ``u = beta u + alpha M f``;
* ``host``: the step through host arrays (page-locked numpy);
* ``dropin``: the reference's own entry points (``create_spme_engine`` /
  ``compute_spme``: host arrays, FP64, reciprocal part);
* ``batch``: many independent systems of uneven size in one step (``Batch``).

Sizes: the benchmark's workloads, the golden vectors' and tests' systems, and
ragged ones at the same density (volume fraction 0.05, mesh spacing about 1.7).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import spme_gb300
from spme_gb300.batch import uneven_systems

XI, RC, RADIUS = 0.3, 10.0, 1.0


def _smooth(n: int) -> int:
    """Smallest 2^a 3^b 5^c >= n."""
    while True:
        m = n
        for q in (2, 3, 5):
            while m % q == 0:
                m //= q
        if m == 1:
            return n
        n += 1


def _box(n: int) -> float:
    """Edge of the box that holds n unit spheres at volume fraction 0.05."""
    return (n * 4.0 / 3.0 * math.pi / 0.05) ** (1.0 / 3.0)


def listed() -> list[dict]:
    return [
        # the smallest system worth a mesh, stepped on the device in a captured loop:
        # launches and latency
        dict(name="tiny_step_fp64", kind="step", N=300, L=32.0, K=32, p=6, R=1, xi=0.5, rc=8.0,
             precision="fp64", graphs=True, tile=""),
        # a program written against the reference: host arrays, FP64, new positions
        # and one force vector per call, BLAS-style accumulation
        dict(name="dropin_n2000", kind="dropin", N=2000, L=50.0, K=64, p=6, R=1, xi=XI, rc=RC,
             precision="fp64", graphs=False, tile=""),
        # a mid-size suspension, one force vector per step, in either precision
        dict(name="single_rhs_fp32", kind="step", N=100_000, L=220.0, K=128, p=6, R=1, xi=XI,
             rc=RC, precision="fp32", graphs=True, tile=""),
        dict(name="single_rhs_fp64", kind="step", N=100_000, L=220.0, K=128, p=6, R=1, xi=XI,
             rc=RC, precision="fp64", graphs=False, tile=""),
        # one iteration of a block Lanczos sampler: fixed positions, eight vectors,
        # low order, a ragged particle count and an odd mesh
        dict(name="lanczos_ragged_fp32", kind="apply", N=20_011, L=119.0, K=75, p=4, R=8, xi=XI,
             rc=RC, precision="fp32", graphs=False, tile=""),
        # high accuracy: FP64, order 8, a few right-hand sides, ragged sizes
        dict(name="multi_rhs_fp64_p8", kind="step", N=30_011, L=136.0, K=90, p=8, R=5, xi=XI,
             rc=RC, precision="fp64", graphs=False, tile=""),
        # an ensemble: 64 independent systems of 500 to 50,000 particles, orders 4, 6, 8
        dict(name="uneven_batch_fp32", kind="batch", count=64, nmin=500, nmax=50_000, R=4, xi=XI,
             rc=RC, precision="fp32", graphs=True, overlap=2),
        # the batched operator: sixteen right-hand sides in one mesh pass
        dict(name="multi_rhs_fp32", kind="step", N=200_000, L=250.0, K=160, p=6, R=16, xi=XI,
             rc=RC, precision="fp32", graphs=False, tile="16x8x4"),
        # ... and the same through host arrays
        dict(name="multi_rhs_host_fp32", kind="host", N=200_000, L=250.0, K=160, p=6, R=16, xi=XI,
             rc=RC, precision="fp32", graphs=False, tile="16x8x4"),
        # a million particles: plain FP64 with one right-hand side, and the FP32 batch
        dict(name="large_fp64", kind="step", N=1_000_000, L=480.0, K=256, p=6, R=1, xi=XI, rc=RC,
             precision="fp64", graphs=False, tile=""),
        dict(name="large_fp32", kind="step", N=1_000_000, L=480.0, K=256, p=6, R=16, xi=XI, rc=RC,
             precision="fp32", graphs=False, tile="16x8x4"),
    ]


def draw(rng: random.Random) -> dict:
    """One more case of the same ranges."""
    kind = rng.choice(["step", "step", "step", "apply", "host", "dropin", "batch"])
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(8, 64), nmin=rng.randint(500, 1000),
                    nmax=rng.randint(8000, 40_000), R=rng.choice([1, 2, 3, 4, 4, 6]), xi=XI, rc=RC,
                    precision=rng.choice(["fp32", "fp32", "fp64"]), graphs=rng.random() < 0.5,
                    overlap=rng.choice([0, 2]))
    precision = "fp64" if kind == "dropin" else rng.choice(["fp32", "fp32", "fp64"])
    top = {"dropin": 30_000, "host": 200_000}.get(kind, 600_000 if precision == "fp32" else 200_000)
    n = int(round(math.exp(rng.uniform(math.log(1500), math.log(top)))))
    L = round(_box(n) * rng.uniform(0.97, 1.05), 2)
    p = rng.choice([4, 6, 6, 8])
    # mostly 5-smooth meshes (odd ones among them), now and then any size
    K = _smooth(int(math.ceil(rng.uniform(0.55, 0.65) * L)))
    if rng.random() < 0.15:
        K = int(math.ceil(0.6 * L))
    R = 1 if kind == "dropin" else rng.choice([1, 1, 2, 3, 4, 7, 8, 12, 16])
    if precision == "fp64":
        R = min(R, 4)
    return dict(kind=kind, N=n, L=L, K=K, p=p, R=R, xi=XI, rc=RC, precision=precision,
                graphs=rng.random() < 0.3, tile=rng.choice(["", "", "16x8x4", "8x8x4"]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

ALPHA, BETA = 0.75, -0.5  # of the kinds that accumulate (apply, dropin)


def _systems(case: dict) -> list[dict]:
    return uneven_systems(count=case["count"], nmin=case["nmin"], nmax=case["nmax"],
                          xi=case["xi"], rc=case["rc"], radius=RADIUS, seed=1234)


def _inputs(case: dict, seed: int) -> dict:
    """Uniform positions, N(0, 1) forces and (for the accumulating kinds) an earlier
    result, on the GPU, from the seed alone."""
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    dt = torch.float32 if case["precision"] == "fp32" else torch.float64
    out = {}
    if case["kind"] == "batch":
        out["systems"] = _systems(case)
        out["pos"] = [torch.rand((s["N"], 3), generator=g, device=dev, dtype=torch.float64) * s["L"]
                      for s in out["systems"]]
        out["f"] = [torch.randn((case["R"], 3 * s["N"]), generator=g, device=dev, dtype=dt)
                    for s in out["systems"]]
        return out
    n, R = case["N"], case["R"]
    out["pos"] = torch.rand((n, 3), generator=g, device=dev, dtype=torch.float64) * case["L"]
    out["f"] = torch.randn((R, 3 * n), generator=g, device=dev, dtype=dt)
    if case["kind"] in ("apply", "dropin"):
        out["u0"] = torch.randn((R, 3 * n), generator=g, device=dev, dtype=dt)
    return out


def prepare(case: dict, seed: int) -> dict:
    x = _inputs(case, seed)
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "batch":
        b = spme_gb300.Batch(x["systems"], nrhs=case["R"], precision=case["precision"])
        b.set_overlap(case["overlap"])
        b.set_graphs(case["graphs"])
        st["batch"] = b
        st["pos"], st["f"] = b.pack(x["pos"]), b.pack(x["f"])
        st["u"] = torch.zeros_like(st["f"])
        return st
    n, L, K, p, R = case["N"], case["L"], case["K"], case["p"], case["R"]
    if kind == "dropin":
        st["handle"] = _Handle(case["xi"], K, p, n, L)
        st["pos"], st["f"], st["u"] = (x[k].cpu().numpy() for k in ("pos", "f", "u0"))
        return st
    tile = tuple(int(t) for t in case["tile"].split("x")) if case["tile"] else None
    e = spme_gb300.Engine(n, L, case["xi"], K, p, radius=RADIUS, rcut=case["rc"],
                          precision=case["precision"], max_nrhs=R, tile=tile)
    e.set_graphs(case["graphs"])
    st["engine"] = e
    if kind == "host":
        st["keep"] = [torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
                      for t in (x["pos"], x["f"], x["f"])]
        st["keep"][0].copy_(x["pos"])
        st["keep"][1].copy_(x["f"])
        st["keep"][2].zero_()
        st["pos"], st["f"], st["u"] = (t.numpy() for t in st["keep"])
        return st
    st["pos"], st["f"] = x["pos"], x["f"]
    st["u"] = x["u0"] if kind == "apply" else torch.zeros_like(x["f"])
    if kind == "apply":
        e.set_positions(st["pos"])
    return st


class _Handle:
    """The reference's engine handle, destroyed with the state that holds it."""

    def __init__(self, xi, dim, porder, n, box):
        self.h = spme_gb300.create_spme_engine(xi, dim, porder, n, box, 1)

    def __del__(self):
        spme_gb300.destroy_spme_engine(self.h)


def run(st: dict):
    kind = st["kind"]
    if kind == "batch":
        return st["batch"].step(st["pos"], st["f"], st["u"])
    if kind == "dropin":
        m = 3 * st["pos"].shape[0]
        spme_gb300.compute_spme(st["handle"].h, st["pos"], st["f"].shape[0], ALPHA, st["f"], m,
                                BETA, st["u"], m)
        return st["u"]
    if kind == "apply":
        return st["engine"].apply(st["f"], st["u"], alpha=ALPHA, beta=BETA)
    st["engine"].set_positions(st["pos"])
    return st["engine"].apply(st["f"], st["u"])


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def _work_one(n, L, K, p, R, rc, elem, real=True, positions=True, accumulate=False):
    C = 3 * R
    nbytes = elem * C * n * (3 if accumulate else 2) + (24 * n if positions else 0)
    # spread and interpolation (one multiply-add per mesh point and component each),
    # two real transforms, the projector (30 real operations per wavevector and
    # right-hand side)
    flops = 2 * 2.0 * p ** 3 * C * n
    flops += 2 * 2.5 * K ** 3 * math.log2(K ** 3) * C
    flops += 30.0 * K * K * (K // 2 + 1) * R
    if real:  # each pair within rc: its two scalar functions, and 18 operations per side
        pairs = n * (n - 1) * 4.0 / 3.0 * math.pi * rc ** 3 / L ** 3
        flops += pairs * (18.0 * R + 25.0)
    return nbytes, flops


def work(case: dict) -> dict:
    elem = 4 if case["precision"] == "fp32" else 8
    kind = case["kind"]
    if kind == "batch":
        parts = [_work_one(s["N"], s["L"], s["K"], s["p"], case["R"], s["rc"], elem)
                 for s in _systems(case)]
        return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}
    b, f = _work_one(case["N"], case["L"], case["K"], case["p"], case["R"], case["rc"], elem,
                     real=kind != "dropin", positions=kind != "apply",
                     accumulate=kind in ("apply", "dropin"))
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the operator in 64 bits
# ---------------------------------------------------------------------------

def _spline(p: int, w):
    """Cardinal B-spline weights M_p(w + p - 1 - j), j = 0 .. p - 1."""
    a = [w, 1.0 - w] + [None] * (p - 2)
    for n in range(3, p + 1):
        b = [None] * p
        b[0] = w * a[0] / (n - 1)
        for k in range(1, n):
            hi = (w + k) * a[k] if k < n - 1 else 0.0
            b[k] = (hi + (n - w - k) * a[k - 1]) / (n - 1)
        a = b
    return a[::-1]


def _recip(pos, L, xi, K, p, f, a=RADIUS):
    """Reciprocal part: spread, transform, influence, transform, interpolate.
    f: (n, C) double, C = 3R.  The index K/2 counts as +K/2 on every axis."""
    dev, C = pos.device, f.shape[1]
    c = torch.remainder(pos, L) * (K / L)
    fl = torch.floor(c)
    start = torch.remainder(fl.long() - p // 2 + 1, K)
    w = [_spline(p, (c - fl)[:, d]) for d in range(3)]
    ix = [[torch.remainder(start[:, d] + j, K) for j in range(p)] for d in range(3)]
    mesh = torch.zeros((K ** 3, C), dtype=torch.float64, device=dev)
    for z in range(p):
        for y in range(p):
            wzy, izy = w[2][z] * w[1][y], (ix[2][z] * K + ix[1][y]) * K
            for x in range(p):
                mesh.index_add_(0, izy + ix[0][x], f * (wzy * w[0][x])[:, None])
    m = torch.arange(K, device=dev)
    kk = torch.where(m <= K // 2, m, m - K).double()
    q = _spline(p, torch.zeros(1, dtype=torch.float64, device=dev))
    ph = 2.0 * math.pi / K * kk
    s = torch.zeros(K, dtype=torch.complex128, device=dev)
    for j in range(p - 1):
        s = s + q[p - 2 - j] * torch.exp(1j * j * ph)
    b2 = 1.0 / (s.real ** 2 + s.imag ** 2)
    k1, Kh = kk * (2.0 * math.pi / L), K // 2 + 1
    kz, ky, kx = k1[:, None, None], k1[None, :, None], k1[None, None, :Kh]
    k2 = kx * kx + ky * ky + kz * kz
    k2[0, 0, 0] = 1.0
    t = k2 / xi ** 2
    tab = 6.0 * math.pi * torch.exp(-t / 4) * (1 - k2 * a * a / 3) / k2 * (1 + t / 4 + t * t / 8)
    tab = tab * (b2[:, None, None] * b2[None, :, None] * b2[None, None, :Kh]) / L ** 3
    tab[0, 0, 0] = 0.0
    neg = torch.remainder(-m, K)
    out = torch.zeros_like(f)
    for r in range(C // 3):
        g = torch.stack([torch.fft.rfftn(mesh[:, 3 * r + d].reshape(K, K, K)) for d in range(3)])
        dot = (kx * g[0] + ky * g[1] + kz * g[2]) / k2
        g[0] -= kx * dot
        g[1] -= ky * dot
        g[2] -= kz * dot
        g *= tab
        for x in [0] + ([K // 2] if K % 2 == 0 else []):  # the part of a real result
            pl = g[:, :, :, x]
            g[:, :, :, x] = 0.5 * (pl + pl[:, neg][:, :, neg].conj())
        for d in range(3):
            mesh[:, 3 * r + d] = (torch.fft.irfftn(g[d], s=(K, K, K)) * float(K) ** 3).reshape(-1)
    for z in range(p):
        for y in range(p):
            wzy, izy = w[2][z] * w[1][y], (ix[2][z] * K + ix[1][y]) * K
            for x in range(p):
                out += mesh[izy + ix[0][x]] * (wzy * w[0][x])[:, None]
    return out


def _pair_functions(r, xi, a):
    """F and G of M_real(r) = F I + G r r^T / r^2: Beenakker's real-space form, and for
    r < 2a the overlap correction, written without its cancelling 1/r terms."""
    rs = 1.0 / math.sqrt(math.pi)
    x = xi * r
    x2 = x * x
    e = torch.exp(-x2) * rs
    near = r < 2 * a
    rn = torch.clamp(r, min=1e-300)
    ec = torch.special.erfc(x)
    far_f = ec * (0.75 / rn + 0.5 * a * a / rn ** 3) + e * (
        4 * xi ** 7 * a * a * r ** 4 + 3 * xi ** 3 * r ** 2 - 20 * xi ** 5 * a * a * r ** 2
        - 4.5 * xi + 14 * xi ** 3 * a * a + xi * a * a / rn ** 2)
    far_g = ec * (0.75 / rn - 1.5 * a * a / rn ** 3) + e * (
        -4 * xi ** 7 * a * a * r ** 4 - 3 * xi ** 3 * r ** 2 + 16 * xi ** 5 * a * a * r ** 2
        + 1.5 * xi - 2 * xi ** 3 * a * a - 3 * xi * a * a / rn ** 2)
    S, P = torch.zeros_like(x), torch.zeros_like(x)
    for n in range(11, -1, -1):  # erf(x)/x and (erf(x) - 2x exp(-x^2)/sqrt(pi))/x^3
        S = S * x2 + 2 * rs * (-1) ** n / (math.factorial(n) * (2 * n + 1))
        P = P * x2 + 2 * rs * (-1) ** n * 2 * (n + 1) / (math.factorial(n + 1) * (2 * n + 3))
    xs = torch.clamp(x, min=0.5)
    ef = torch.special.erf(xs)
    small = x < 0.5
    S = torch.where(small, S, ef / xs)
    P = torch.where(small, P, (ef - 2 * xs * e) / xs ** 3)
    x4, c = x2 * x2, xi ** 3 * a * a
    near_f = xi * (-0.75 * S + e * (3 * x2 - 4.5)) + c * (
        -0.5 * P + e * (4 * x4 - 20 * x2 + 14)) + (1 - 9 * r / (32 * a)) / a
    near_g = xi * (-0.75 * S + e * (1.5 - 3 * x2)) + c * (
        1.5 * P + e * (-4 * x4 + 16 * x2 - 2)) + 3 * r / (32 * a * a)
    return torch.where(near, near_f, far_f), torch.where(near, near_g, far_g)


def _real_self(pos, L, xi, rc, f, a=RADIUS):
    """Pairs within rc (minimum image) and the self term."""
    n, dev = pos.shape[0], pos.device
    rs = 1.0 / math.sqrt(math.pi)
    out = f * ((1 - 6 * xi * a * rs + 40.0 / 3.0 * (xi * a) ** 3 * rs) / a)
    x = torch.remainder(pos, L)
    nc = int(L / rc)
    if nc < 3:
        nc = 1
    nc = min(nc, 100)
    cell3 = torch.clamp((x * (nc / L)).long(), max=nc - 1)
    cell = (cell3[:, 2] * nc + cell3[:, 1]) * nc + cell3[:, 0]
    order = torch.argsort(cell)
    x, cell3, fs = x[order], cell3[order], f[order]
    count = torch.bincount(cell, minlength=nc ** 3)
    first = torch.cumsum(count, 0) - count
    most = int(count.max())
    me = torch.arange(n, device=dev)
    acc = torch.zeros_like(f)
    span = (-1, 0, 1) if nc > 1 else (0,)
    for dz in span:
        for dy in span:
            for dx in span:
                o = [torch.remainder(cell3[:, d] + s, nc) for d, s in enumerate((dx, dy, dz))]
                c2 = (o[2] * nc + o[1]) * nc + o[0]
                beg, cnt = first[c2], count[c2]
                for t in range(most):
                    i = torch.nonzero((cnt > t) & (beg + t != me)).squeeze(1)
                    j = beg[i] + t
                    d = x[i] - x[j]
                    d -= L * torch.round(d / L)
                    r2 = (d * d).sum(1)
                    keep = torch.nonzero(r2 < rc * rc).squeeze(1)
                    i, j, d, r = i[keep], j[keep], d[keep], torch.sqrt(r2[keep])
                    F, G = _pair_functions(r, xi, a)
                    d = d / torch.clamp(r, min=1e-300)[:, None]
                    fj = fs[j].reshape(len(i), f.shape[1] // 3, 3)
                    dot = (fj * d[:, None, :]).sum(2, keepdim=True)
                    add = F[:, None, None] * fj + G[:, None, None] * dot * d[:, None, :]
                    acc.index_add_(0, i, add.reshape(len(i), f.shape[1]))
    res = torch.empty_like(acc)
    res[order] = acc
    return out + res


def _mobility(pos, L, xi, rc, K, p, f, real=True):
    """(R, 3n) -> (R, 3n)."""
    R, n = f.shape[0], pos.shape[0]
    rows = f.double().reshape(R, n, 3).transpose(0, 1).reshape(n, 3 * R).contiguous()
    u = _recip(pos, L, xi, K, p, rows)
    if real:
        u = u + _real_self(pos, L, xi, rc, rows)
    return u.reshape(n, R, 3).transpose(0, 1).reshape(R, 3 * n)


def exact(case: dict, seed: int):
    x = _inputs(case, seed)
    if case["kind"] == "batch":
        return torch.cat([_mobility(q, s["L"], s["xi"], s["rc"], s["K"], s["p"], f).reshape(-1)
                          for s, q, f in zip(x["systems"], x["pos"], x["f"])])
    u = _mobility(x["pos"], case["L"], case["xi"], case["rc"], case["K"], case["p"], x["f"],
                  real=case["kind"] != "dropin")
    if "u0" in x:
        u = ALPHA * u + BETA * x["u0"].double()
    return u.cpu().numpy() if case["kind"] in ("dropin", "host") else u
