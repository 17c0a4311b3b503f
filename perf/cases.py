"""The solver's work that is measured: its cases, their inputs, one pass of each
through the public API, and what the pass has to come to in 64 bits.

A case names a kind of work and its sizes:

* ``solve``     -- SolvePDE of a Fourier x GLL plan (2D or 3D, one or several GLL
  elements, Dirichlet or Robin ends, or periodic in the GLL direction as well;
  the stock operator or the caller's own)
* ``misfit``    -- SolvePDE and the gradient of a least-squares loss
  (SolveAdjointMisfit), as an inversion step calls them
* ``autograd``  -- helmholtz_solve inside a torch graph, and its backward pass
* ``batch``     -- many independent 2D problems of uneven sizes in one call
* ``fd``        -- the finite-difference solver, alone or with its gradient
* ``derivs``    -- the first or second derivatives of a field in every direction

``Nx`` (by ``Ny``, 0 in 2D) is the Fourier grid, ``N`` the GLL points of an element (the interior points in
z of a finite-difference grid), ``Ns`` the elements.  ``bc`` holds the Robin
coefficients by name, ``io`` the bytes of f and u.
"""
import math

import numpy as np
import torch

from mpi_b200 import (BatchNonPeriodic2D, Helmholtz3DFD, NonPeriodic2D, NonPeriodic3D, Periodic2D, Periodic3D)
from mpi_b200.autograd import helmholtz_solve

LX, LY, LZ = 2.0 * math.pi, 2.0 * math.pi, 2.0

# alpha, beta at the lower end, alpha, beta at the upper end
ENDS = {"dirichlet": (0.0, 1.0, 0.0, 1.0), "neumann_dirichlet": (1.0, 0.0, 0.0, 1.0), "robin": (1.0, 0.5, 0.7, 2.0)}


def _case(kind, Nx, Ny, N, Ns=1, bc="dirichlet", lam=1.0, precision="fp64", **more):
    c = {"kind": kind, "Nx": Nx, "Ny": Ny, "N": N, "Ns": Ns, "bc": bc, "lam": lam, "precision": precision}
    c.update(more)
    return c


def listed():
    cases = []

    def add(name, *a, **k):
        cases.append(dict(_case(*a, **k), name=name))

    # the smallest call: one 64 x 33 problem with Dirichlet ends, where latency is all there is
    add("solve2d_64x33", "solve", 64, 0, 33)
    # the stock 2D problem: 52 elements of 10 points, Neumann below, Dirichlet above, boundary data
    add("solve2d_512x10_52el", "solve", 512, 0, 10, 52, "neumann_dirichlet")
    # the stock 3D problem periodic in every direction: 25 elements of 10 points
    add("periodic3d_64x32x10_25el", "solve", 64, 32, 10, 25, "periodic")
    # a caller's own operator with a coefficient that varies in z: a factor of its own per wavenumber pair
    add("operator3d_64x32x33", "solve", 64, 32, 33, operator=True)
    # one element of an even, ragged number of points, Robin ends with data, unequal x and y
    add("robin3d_64x128x50", "solve", 64, 128, 50, 1, "robin")
    # the benchmark's own problem, at the precision that it reports
    add("solve3d_256x256x65_refine", "solve", 256, 256, 65, lam=10.0, precision="fp32_refine")
    # an inversion step in FP32: forward solve, gradient of the misfit in f and lambda
    add("misfit3d_128x128x65_fp32", "misfit", 128, 128, 65, lam=5.0, precision="fp32")
    # the differentiable solve in a torch graph, several elements, gradients of every input
    add("autograd3d_64x32x17_4el", "autograd", 64, 32, 17, 4, "robin", lam=2.0)
    # 512 problems of uneven sizes in one call
    add("batch2d_512", "batch", 512, 0, 0, precision="fp32_refine", count=512)
    # the largest: finite differences on 1024 x 1024 x 256 points
    add("fd3d_1024x1024x256", "fd", 1024, 1024, 256)
    # a refined finite-difference inversion step, Robin ends, a ragged number of points in z
    add("fd3d_misfit_256x128x100_refine", "fd", 256, 128, 100, 1, "robin", precision="fp32_refine", gradient=True)
    # d/dx, d/dy, d/dz of a field: what a time stepper or a residual asks for
    add("derivs3d_256x256x65", "derivs", 256, 256, 65, order=1)
    return cases


def _pow2(rng, lo, hi):
    return 1 << rng.randint(lo.bit_length() - 1, hi.bit_length() - 1)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "misfit", "autograd", "batch", "fd", "fd", "derivs"])
    lam = round(10.0 ** rng.uniform(-1.0, 2.0), 4)
    if kind == "batch":
        return _case("batch", 512, 0, 0, lam=lam, precision=rng.choice(["fp64", "fp32_refine"]),
                     count=_log(rng, 8, 512))
    if kind == "fd":
        while True:
            Nx, Ny, Nz = _pow2(rng, 32, 512), _pow2(rng, 32, 512), _log(rng, 9, 500)
            if Nx * Ny * Nz <= 1 << 25:  # with sweeps and a gradient no dearer than the largest listed case
                break
        c = _case("fd", Nx, Ny, Nz, 1, rng.choice(["dirichlet", "robin", "neumann_dirichlet"]), lam,
                  rng.choice(["fp64", "fp32", "fp32_refine"]))
        c["gradient"] = rng.random() < 0.4
        if c["precision"] == "fp32":
            # FP32 is used where the stencil's condition, about (Nz / pi)^2 / lambda, leaves it enough digits
            c.update(N=min(Nz, 64), lam=max(lam, 20.0), gradient=False, io=4)
        return c
    three = kind != "solve" or rng.random() < 0.6
    precision = rng.choice(["fp64", "fp64", "fp32", "fp32_refine"])
    while True:
        Nx = _pow2(rng, 16, 256) if three else _pow2(rng, 16, 1024)
        Ny = _pow2(rng, 16, 256) if three else 0
        Ns = rng.choice([1, 1, _log(rng, 2, 60)])
        N = _log(rng, 5, 129) if Ns == 1 else _log(rng, 5, 33)
        # no more points than the benchmark's problem, and a dense 64-bit solve that stays quick
        if Nx * max(1, Ny) * N * Ns <= 256 * 256 * 65 and Ns * N <= 640:
            break
    bc = rng.choice(["dirichlet", "robin", "neumann_dirichlet", "periodic"])
    if kind == "autograd" or (kind == "misfit" and Ns > 1):
        bc = rng.choice(["dirichlet", "robin", "neumann_dirichlet"])
    c = _case(kind, Nx, Ny, N, Ns, bc, lam, precision)
    if kind == "derivs":
        c["order"] = rng.choice([1, 2])
        c["precision"] = rng.choice(["fp64", "fp64", "fp32"])
    if c["precision"] == "fp32":
        # as above: one element, ends without slopes, first derivatives
        c.update(N=min(N, 66), Ns=1, bc="dirichlet")
        if kind == "derivs":
            c["order"] = 1
        if kind in ("solve", "derivs"):
            c["io"] = 4
    if kind == "solve" and c["precision"] != "fp32_refine" and c["N"] <= 65 and Nx * max(1, Ny) <= 4096 \
            and rng.random() < 0.25:
        c["operator"] = True
    return c


# ------------------------------------------------------------------- inputs --
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gll(N):
    """GLL nodes on [-1, 1] and their first-derivative matrix."""
    leg = np.polynomial.legendre
    c = np.zeros(N)
    c[-1] = 1.0
    x = np.sort(leg.legroots(leg.legder(c)).real)
    for _ in range(3):  # Newton on P'_{N-1}
        x = x - leg.legval(x, leg.legder(c)) / leg.legval(x, leg.legder(c, 2))
    x = 0.5 * (x - x[::-1])
    x = np.concatenate(([-1.0], x, [1.0]))
    p = leg.legval(x, c)
    diff = x[:, None] - x[None, :] + np.eye(N)
    D = p[:, None] / (p[None, :] * diff)
    np.fill_diagonal(D, 0.0)
    D[0, 0], D[-1, -1] = -N * (N - 1) / 4.0, N * (N - 1) / 4.0
    return x, D


def _nodes(case):
    """[Ns, N] positions along the last direction, mapped to [-1, 1]."""
    N, Ns = case["N"], case["Ns"]
    if case["kind"] == "fd":
        return (2.0 * np.arange(1, N + 1) / (N + 1) - 1.0)[None, :]
    x, _ = _gll(N)
    return np.stack([(2.0 * j + 1.0 + x) / Ns - 1.0 for j in range(Ns)])


def _smooth(case, gen, dev):
    """A smooth random field [Ns, Nx, (Ny,) N]: Fourier modes in x and y times
    Chebyshev polynomials along the last direction (cosines where that is
    periodic), amplitudes (1 + |k|^2)^-1.5."""
    Nx, Ny = case["Nx"], max(1, case["Ny"])
    t = torch.from_numpy(_nodes(case)).to(dev)
    nl = min(case["N"] * case["Ns"], 24)
    l = torch.arange(nl, dtype=torch.float64, device=dev)
    angle = math.pi * (t + 1.0) if case["bc"] == "periodic" else torch.acos(t.clamp(-1.0, 1.0))
    basis = torch.cos(l[:, None, None] * angle)
    kx = torch.fft.fftfreq(Nx, 1.0 / Nx, dtype=torch.float64, device=dev)
    ky = torch.fft.rfftfreq(Ny, 1.0 / Ny, dtype=torch.float64, device=dev)
    amp = (1.0 + kx[:, None, None] ** 2 + ky[None, :, None] ** 2 + l ** 2) ** -1.5
    shape = tuple(amp.shape)
    co = torch.complex(torch.randn(shape, generator=gen, dtype=torch.float64, device=dev),
                       torch.randn(shape, generator=gen, dtype=torch.float64, device=dev)) * amp
    plane = torch.fft.irfft2(co, s=(Nx, Ny), dim=(0, 1)) * (Nx * Ny)
    out = torch.matmul(plane.reshape(Nx * Ny, nl), basis.reshape(nl, -1))
    out = out.reshape(Nx, Ny, case["Ns"], case["N"]).permute(2, 0, 1, 3).contiguous()
    return out if case["Ny"] else out[:, :, 0].contiguous()


def _batch_sizes(case, seed):
    rng = np.random.default_rng(seed)
    n = case["count"]
    Nx = [int(v) for v in rng.choice((32, 64, 128, 256, 512), n)]
    P = [int(v) + 1 for v in rng.choice((16, 32, 64, 128), n)]
    lam = [float(v) for v in 10.0 ** rng.uniform(-2.0, 4.0, n)]
    return Nx, P, lam


def _inputs(case, seed):
    """f, boundary data and the observed field, from the seed alone."""
    dev = _device()
    gen = torch.Generator(device=dev).manual_seed(seed)
    if case["kind"] == "batch":
        # the sizes belong to the program, the right-hand sides to the seed
        Nx, P, _ = _batch_sizes(case, case["count"])
        return {"f": [_smooth(_case("solve", a, 0, p), gen, dev)[0] for a, p in zip(Nx, P)]}
    s = {"f": _smooth(case, gen, dev)}
    g = (case["Nx"], case["Ny"]) if case["Ny"] else (case["Nx"],)
    # Dirichlet solves run without data (zero ends); Robin ends come with theirs
    if case["bc"] not in ("dirichlet", "periodic") or case["kind"] == "autograd":
        s["gl"] = torch.randn(g, generator=gen, dtype=torch.float64, device=dev)
        s["gr"] = torch.randn(g, generator=gen, dtype=torch.float64, device=dev)
    if case["kind"] in ("misfit", "autograd") or case.get("gradient"):
        s["obs"] = 0.1 * _smooth(case, gen, dev)
    if case.get("io") == 4:
        s["f"] = s["f"].float()
    return s


def _coefficient(case):
    """c(z) of a caller's own operator d2/dz2 - (sigma + c(z)), at the interior nodes."""
    x, _ = _gll(case["N"])
    return 1.0 + 0.5 * np.sin(2.0 * x[1:-1])


def _plan(case):
    Nx, Ny, N, Ns, p = case["Nx"], case["Ny"], case["N"], case["Ns"], case["precision"]
    k = {"Lambda": case["lam"], "precision": p}
    box = (0.0, LX, 0.0, LY, 0.0, LZ) if Ny else (0.0, LX, 0.0, LZ)
    if case["kind"] == "fd":
        plan = Helmholtz3DFD(Nx, Ny, N, *box, bc=ENDS[case["bc"]], **k)
    elif case["bc"] == "periodic":
        plan = Periodic3D(Nx, Ny, N * Ns, N, *box, **k) if Ny else Periodic2D(Nx, N * Ns, N, *box, **k)
    else:
        k["bc"] = ENDS[case["bc"]]
        plan = NonPeriodic3D(Nx, Ny, N * Ns, N, *box, **k) if Ny else NonPeriodic2D(Nx, N * Ns, N, *box, **k)
    if case.get("operator"):
        # the interior operator of every wavenumber pair, as the caller builds it from the plan's grid
        _, _, D2 = plan.grid()
        base = D2.numpy()[1:-1, 1:-1] - np.diag(_coefficient(case))
        eye = np.eye(N - 2)
        plan.SetOperator(lambda iw, jw: base - (case["lam"] + (2 * math.pi * iw / LX) ** 2
                                                + (2 * math.pi * jw / LY) ** 2) * eye)
    if case.get("io") == 4:
        plan.set_io_bytes(4)
    return plan


def prepare(case, seed):
    s = _inputs(case, seed)
    s["kind"], s["bc"], s["gradient"], s["order"] = (case["kind"], case["bc"], case.get("gradient", False),
                                                     case.get("order", 1))
    s["floats"] = case["precision"] == "fp32"
    if case["kind"] == "batch":
        Nx, P, lam = _batch_sizes(case, case["count"])
        s["plan"] = BatchNonPeriodic2D(Nx, P, lam, 0.0, LX, 0.0, LZ, precision=case["precision"])
        s["f"] = s["plan"].pack(s["f"])
        return s
    s["plan"] = _plan(case)
    if case["kind"] == "autograd":
        s["lam"] = torch.tensor(case["lam"], dtype=torch.float64, device=s["f"].device, requires_grad=True)
        for k in ("f", "gl", "gr"):
            s[k].requires_grad_(True)
    return s


# ----------------------------------------------------------------- one pass --
def run(s):
    plan, f, kind = s["plan"], s["f"], s["kind"]
    if kind == "batch":
        return plan.solve(f)
    if kind == "derivs":
        if f.dim() == 4:
            if s["order"] == 1:
                return plan.FirstDerivativeX(f), plan.FirstDerivativeY(f), plan.FirstDerivativeZ(f)
            return plan.SecondDerivativeX(f), plan.SecondDerivativeY(f), plan.SecondDerivativeZ(f)
        if s["order"] == 1:
            return plan.FirstDerivativeX(f), plan.FirstDerivativeY(f)
        return plan.SecondDerivativeX(f), plan.SecondDerivativeY(f)
    if kind == "autograd":
        u = helmholtz_solve(plan, f, s["lam"], s["gl"], s["gr"])
        loss = 0.5 * ((u - s["obs"]) ** 2).sum()
        got = (u.detach(),) + torch.autograd.grad(loss, (f, s["lam"], s["gl"], s["gr"]))
        return tuple(t.float() for t in got) if s["floats"] else got
    if s["bc"] == "periodic":
        u = plan.SolvePDE(f)
    else:
        u = plan.SolvePDE(f, s.get("gl"), s.get("gr"))
    if kind == "misfit" or s["gradient"]:
        fbar, lbar, _, _ = plan.SolveAdjointMisfit(u, s["obs"])
        return (u.float(), fbar.float(), lbar.float()) if s["floats"] else (u, fbar, lbar)
    return u


# --------------------------------------------------------------------- work --
def work(case):
    """Every input read and every output written once; the transforms' and the
    row solves' operations."""
    if case["kind"] == "batch":
        Nx, P, _ = _batch_sizes(case, case["count"])
        pts = sum(a * p for a, p in zip(Nx, P))
        return {"bytes": 16.0 * pts,
                "flops": float(sum(5 * a * p * math.log2(a) + 2 * a * p * p for a, p in zip(Nx, P)))}
    Nx, Ny, N, Ns = case["Nx"], case["Ny"], case["N"], case["Ns"]
    pts = float(Nx * max(1, Ny) * N * Ns)
    data = 16.0 * Nx * max(1, Ny) if case["bc"] not in ("dirichlet", "periodic") else 0.0
    lg = math.log2(Nx) + (math.log2(Ny) if Ny else 0.0)
    io = float(case.get("io", 8))
    if case["kind"] == "derivs":
        # the field once, its derivatives once each
        return {"bytes": pts * io * (4 if Ny else 3), "flops": pts * (5 * lg + 2 * N)}
    row = 16.0 if case["kind"] == "fd" else 2.0 * N
    one = {"bytes": 2 * pts * io + data, "flops": pts * (5 * lg + row)}
    if case["kind"] in ("misfit", "autograd") or case.get("gradient"):
        # f, the observed field and u in; u and the gradient of f out (the loss reads u)
        one = {"bytes": pts * 8 * 5 + 2 * data, "flops": 2 * one["flops"] + 3 * pts}
    return one


# -------------------------------------------------------------------- exact --
def _exact_rows(case, fh, glh, grh, lam):
    """Solutions of every wavenumber pair: fh [nk, Ns, N, m], glh / grh [nk, m]
    (real, m right-hand sides a pair shares), sigma [nk] -> [nk, Ns, N, m]."""
    N, Ns = case["N"], case["Ns"]
    dev = fh.device
    _, D = _gll(N)
    h = 2.0 * Ns / LZ
    D = torch.from_numpy(D * h).to(dev)
    D2 = D @ D
    per = case["bc"] == "periodic"
    K = Ns * (N - 1) + (0 if per else 1)
    base = torch.zeros(K, K, dtype=torch.float64, device=dev)
    inner = torch.zeros(K, dtype=torch.float64, device=dev)
    where = torch.tensor([[(j * (N - 1) + i) % K for i in range(N)] for j in range(Ns)], device=dev)
    for j in range(Ns):
        at = where[j]
        rows = at[1:-1]
        base[rows[:, None], at[None, :]] += D2[1:-1]
        if case.get("operator"):
            base[rows, rows] -= torch.from_numpy(_coefficient(case)).to(dev)
        inner[rows] = 1.0
        nxt = (j + 1) % Ns
        if per or j + 1 < Ns:  # equal slopes where two elements meet
            meet = ((j + 1) * (N - 1)) % K
            base[meet].index_add_(0, at, D[-1])
            base[meet].index_add_(0, where[nxt], -D[0])
    if not per:
        al, bl, ar, br = ENDS[case["bc"]]
        base[0].index_add_(0, where[0], -al * D[0])
        base[0, 0] += bl
        base[K - 1].index_add_(0, where[-1], ar * D[-1])
        base[K - 1, K - 1] += br
    rhs = torch.zeros(fh.shape[0], K, fh.shape[-1], dtype=torch.float64, device=dev)
    rhs = rhs.index_copy(1, where[:, 1:-1].reshape(-1), fh[:, :, 1:-1].reshape(fh.shape[0], -1, fh.shape[-1]))
    if not per and glh is not None:
        rhs = rhs.index_copy(1, torch.tensor([0, K - 1], device=dev), torch.stack([glh, grh], 1))
    out = []
    step = max(1, int(2.0e8 / (K * K)))
    for i in range(0, rhs.shape[0], step):
        M = base - lam[i:i + step, None, None] * torch.diag(inner)
        out.append(torch.linalg.solve(M, rhs[i:i + step]))
    return torch.cat(out)[:, where.reshape(-1)].reshape(rhs.shape[0], Ns, N, -1)


def _exact_solve(case, f, gl, gr, lam):
    """u of one forward solve in 64 bits, differentiable in f, gl, gr and lam."""
    Nx, Ny, N, Ns = case["Nx"], case["Ny"], case["N"], case["Ns"]
    ny = max(1, Ny)
    dev = f.device
    f = f.reshape(Ns, Nx, ny, N)
    fh = torch.fft.fft(torch.fft.rfft(f, dim=1), dim=2)
    nk = Nx // 2 + 1
    half = ny // 2 + 1
    # wavenumbers ky and -ky share an operator
    ky = torch.arange(half, device=dev)
    pair = torch.stack([ky, (ny - ky) % ny], 1)

    def gather(a):  # [nk, ny, ...] complex -> [nk * half, ..., 4] real
        a = a[:, pair]
        a = torch.view_as_real(a).movedim(2, -2)
        return a.reshape(nk * half, *a.shape[2:-2], 4)

    def bc(g):
        return gather(torch.fft.fft(torch.fft.rfft(g.reshape(Nx, ny), dim=0), dim=1)) if g is not None else None

    kx = torch.arange(nk, dtype=torch.float64, device=dev)
    sig = lam + ((2 * math.pi / LX * kx[:, None]) ** 2 + (2 * math.pi / LY * ky.double()[None, :]) ** 2).reshape(-1)
    x = _exact_rows(case, gather(fh.movedim(0, 2)), bc(gl), bc(gr), sig)
    x = torch.view_as_complex(x.reshape(nk, half, Ns, N, 2, 2).contiguous())
    full = torch.cat([x[:, :, :, :, 0], x[:, 1:ny - half + 1, :, :, 1].flip(1)], 1).movedim(2, 0)
    u = torch.fft.irfft(torch.fft.ifft(full, dim=2), n=Nx, dim=1)
    return u.reshape((Ns, Nx, Ny, N) if Ny else (Ns, Nx, N))


def _exact_fd(case, f, gl, gr, lam):
    """The finite-difference solve in 64 bits: transforms in x and y, one
    tridiagonal elimination along z of all wavenumbers at once."""
    Nx, Ny, Nz = case["Nx"], case["Ny"], case["N"]
    dev = f.device
    fh = torch.fft.rfft2(f.reshape(Nx, Ny, Nz), dim=(0, 1))
    dx, dy, dz = LX / Nx, LY / Ny, LZ / (Nz + 1)
    cz = 1.0 / dz ** 2
    al, bl, ar, br = ENDS[case["bc"]]
    a0, a1, a2 = 1.5 * al / dz + bl, -2.0 * al / dz, 0.5 * al / dz
    e0, e1, e2 = 1.5 * ar / dz + br, -2.0 * ar / dz, 0.5 * ar / dz
    kx = torch.arange(Nx, dtype=torch.float64, device=dev)
    ky = torch.arange(Ny // 2 + 1, dtype=torch.float64, device=dev)
    shift = (lam + (4.0 / dx ** 2 * torch.sin(math.pi * kx / Nx) ** 2)[:, None]
             + (4.0 / dy ** 2 * torch.sin(math.pi * ky / Ny) ** 2)[None, :])
    dia = -2.0 * cz - shift
    sup0, subn = cz - cz * a2 / a0, cz - cz * e2 / e0
    cs, ds = [], []
    for k in range(Nz):
        b = dia - (cz * a1 / a0 if k == 0 else cz * e1 / e0 if k == Nz - 1 else 0.0)
        r = fh[..., k]
        if k == 0 and gl is not None:
            r = r - cz / a0 * torch.fft.rfft2(gl)
        if k == Nz - 1 and gr is not None:
            r = r - cz / e0 * torch.fft.rfft2(gr)
        if k:
            a = subn if k == Nz - 1 else cz
            b = b - a * cs[-1]
            r = r - a * ds[-1]
        cs.append((sup0 if k == 0 else cz) / b)
        ds.append(r / b)
    x = [ds[-1]]
    for k in range(Nz - 2, -1, -1):
        x.append(ds[k] - cs[k] * x[-1])
    del fh, cs, ds
    u = torch.fft.irfft2(torch.stack(x[::-1], -1), s=(Nx, Ny), dim=(0, 1))
    return u.reshape(1, Nx, Ny, Nz)


def _exact_derivs(case, f):
    Nx, Ny, N, Ns, order = case["Nx"], case["Ny"], case["N"], case["Ns"], case["order"]
    f = f.double()

    def fourier(dim, n, L):
        k = torch.fft.rfftfreq(n, 1.0 / n, dtype=torch.float64, device=f.device)
        m = (2j * math.pi / L * k) ** order
        if order == 1:
            m[-1] = 0.0
        shape = [1] * f.dim()
        shape[dim] = -1
        return torch.fft.irfft(torch.fft.rfft(f, dim=dim) * m.reshape(shape), n=n, dim=dim)

    _, D = _gll(N)
    D = torch.from_numpy(D * (2.0 * Ns / LZ)).to(f.device)
    M = D if order == 1 else D @ D
    out = [fourier(1, Nx, LX)] + ([fourier(2, Ny, LY)] if Ny else [])
    return tuple(out) + (f @ M.T,)


def exact(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    if kind == "batch":
        Nx, P, lam = _batch_sizes(case, case["count"])
        out = [None] * len(Nx)
        for key in sorted(set(zip(Nx, P))):
            c = _case("solve", key[0], 0, key[1])
            for i in [i for i, k in enumerate(zip(Nx, P)) if k == key]:
                out[i] = _exact_solve(c, s["f"][i], None, None, lam[i]).reshape(-1)
        return torch.cat(out)
    if kind == "derivs":
        return _exact_derivs(case, s["f"])
    f = s["f"].double()
    lam = torch.tensor(case["lam"], dtype=torch.float64, device=f.device)
    solve = _exact_fd if kind == "fd" else _exact_solve
    gl, gr = s.get("gl"), s.get("gr")
    if "obs" not in s:
        return solve(case, f, gl, gr, lam)
    if case["Nx"] * case["Ny"] * case["N"] > 1 << 23:
        return None  # the graph of the elimination would not be quick
    want = [f, lam] + ([gl, gr] if kind == "autograd" else [])
    for t in want:
        t.requires_grad_(True)
    u = solve(case, f, gl, gr, lam)
    g = torch.autograd.grad(0.5 * ((u - s["obs"]) ** 2).sum(), want)
    if kind == "autograd":
        return (u.detach(),) + g
    return u.detach(), g[0], g[1].reshape(1)
