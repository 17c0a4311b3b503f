"""Row solves of several GLL elements of more than 34 points (multi_rows_kernel with
all of a CTA's warps on each vector): the compiled kernels keep their accumulators in
registers; on the GPU the edges of the product tiles, of the 16-vector rounds and of
the largest elements against the oracle, the adjoint through the dot-product
identity."""
import os
import re
import subprocess

import numpy as np
import pytest
import torch

from mpi_b200 import NonPeriodic2D, NonPeriodic3D, Periodic2D
from mpi_b200 import build as B
from oracle import oracle as O
from tests.helpers import rel_l2


def test_row_kernels_keep_their_accumulators_in_registers(tmp_path):
    cmd = [B.NVCC] + B.ARCH + B.COMMON + ["-Xptxas", "-v", "-c", os.path.join(B.CSRC, "helm_multi.cu"), "-o",
                                          str(tmp_path / "multi.o")]
    log = subprocess.run(cmd, capture_output=True, text=True, check=True).stderr
    spills = [int(v) for v in re.findall(r"(\d+) bytes spill stores", log)]
    assert len(spills) >= 16  # a kernel per precision, size class and direction
    # two values at most: whole-row accumulators that do not fit take hundreds of bytes
    assert max(spills) <= 16


# (Nx, Ny, N, Ns).  n = N - 2 interior points: 32 (the last size with a warp's own
# accumulators), 33; 38, 39, 40 (the two end-slope rows begin a tile at 39 and 40);
# 48; the largest, 119 .. 127, whose slope rows cross a tile at 119, 120, 126 and 127.
# Vectors per CTA: 2 and 3 (part of a group), 16, 17 and 40 (one, two and three
# rounds), and several rows per CTA in 3D with a last CTA of fewer rows
SHAPES = [(8, 0, 34, 2), (8, 0, 35, 2), (8, 0, 40, 3), (8, 0, 41, 16), (8, 0, 42, 17), (4, 0, 50, 40), (8, 0, 67, 3),
          (8, 0, 103, 2), (32, 64, 36, 2)]
LARGEST = [(8, 0, 121, 2), (8, 0, 122, 3), (4, 0, 128, 2), (4, 0, 129, 5)]
CASES = [(s, p) for s in SHAPES for p in ("fp64", "fp32", "fp32_refine")] + [(s, "fp32") for s in LARGEST]
BC = (1.0, 0.5, 0.7, 2.0)


def _tol(N, Ns, precision):
    # FP64: eps times the condition of the chain of elements, whose largest eigenvalue
    # is about 0.1 N^4 Ns^2 times its smallest; FP32: about 100 eps_32, and the rounding of
    # the D-weighted right-hand sides, which grow with N^2, beyond 100 points
    return 2.2e-16 * 0.1 * N**4 * Ns**2 + 1e-13 if precision != "fp32" else 1e-5 * max(1.0, (N / 100.0) ** 2)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("shape,precision", CASES)
def test_forward_and_adjoint(cuda, shape, precision):
    Nx, Ny, N, Ns = shape
    rng = np.random.default_rng(N * Ns)
    g = (Nx, Ny) if Ny else (Nx,)
    f, gl, gr = rng.standard_normal((Ns,) + g + (N,)), rng.standard_normal(g), rng.standard_normal(g)
    lam = 3.0
    if Ny:
        ref = O.solve3d(f, gl, gr, Lx=1.3, Ly=0.8, Lz=0.9, lam=lam, bc=BC)
        p = NonPeriodic3D(Nx, Ny, Ns * N, N, 0.0, 1.3, 0.0, 0.8, 0.0, 0.9, Lambda=lam, bc=BC, precision=precision)
    else:
        ref = O.solve2d(f, gl, gr, Lx=1.3, Ly=0.9, lam=lam, bc=BC)
        p = NonPeriodic2D(Nx, Ns * N, N, 0.0, 1.3, 0.0, 0.9, Lambda=lam, bc=BC, precision=precision)
    assert "multi_rows_kernel" in p.kernels()
    tol = _tol(N, Ns, precision)
    u = p.SolvePDE(_dev(f), _dev(gl), _dev(gr))
    assert rel_l2(u.cpu().numpy(), ref) < tol
    ubar = rng.standard_normal(f.shape)
    fbar, _, glb, grb = p.SolveAdjoint(_dev(ubar), u=_dev(ref), want_bc=True)
    fb, a, b = fbar.cpu().numpy(), glb.cpu().numpy(), grb.cpu().numpy()
    lhs = float((ref * ubar).sum())
    rhs = float((f * fb).sum() + (gl * a).sum() + (gr * b).sum())
    # each side's rounding is relative to the products it sums
    scale = np.linalg.norm(ref) * np.linalg.norm(ubar) + np.linalg.norm(f) * np.linalg.norm(fb) \
        + np.linalg.norm(gl) * np.linalg.norm(a) + np.linalg.norm(gr) * np.linalg.norm(b)
    assert abs(lhs - rhs) < tol * scale


@pytest.mark.gpu
@pytest.mark.parametrize("shape,precision", [(s, p) for s, p in CASES if not s[1]])
def test_periodic(cuda, shape, precision):
    Nx, _, N, Ns = shape
    f = np.random.default_rng(N + Ns).standard_normal((Ns, Nx, N))
    ref = O.psolve2d(f, Lx=1.3, Ly=0.9, lam=3.0)
    p = Periodic2D(Nx, Ns * N, N, 0.0, 1.3, 0.0, 0.9, Lambda=3.0, precision=precision)
    assert "multi_rows_kernel" in p.kernels()
    assert rel_l2(p.SolvePDE(_dev(f)).cpu().numpy(), ref) < _tol(N, Ns, precision)
