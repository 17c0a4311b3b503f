"""Row solves of plans with several GLL elements (multi_rows_kernel): every
tile edge of its products, few and many elements, ragged last CTAs, against the
oracle; the adjoint through the dot-product identity with the oracle's map."""
import numpy as np
import pytest
import torch

from mpi_b200 import NonPeriodic2D, NonPeriodic3D, Periodic2D
from oracle import oracle as O
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# (Nx, Ny, N, Ns): one interior point; n = 7, 8, 9, 15, 16, 17 about the 8-wide
# tiles (and n + 2 about the next); n = 62, 64, 98; 64 elements; two rows per
# CTA with a last CTA of one row (513 rows); several rows per CTA in 3D
SHAPES = [(8, 0, 3, 2), (8, 0, 9, 3), (8, 0, 10, 2), (16, 0, 11, 5), (8, 0, 17, 2), (8, 0, 18, 4), (8, 0, 19, 3),
          (8, 0, 64, 2), (4, 0, 66, 2), (4, 0, 100, 3), (16, 0, 5, 64), (1024, 0, 5, 2), (16, 128, 6, 3)]
BCS = [(0.0, 1.0, 0.0, 1.0), (1.0, 0.5, 0.7, 2.0)]


def _tol(N, Ns, precision):
    # FP64: eps times the condition of the chain of elements, whose largest
    # eigenvalue is about 0.1 N^4 Ns^2 times its smallest; FP32: the spectrum's
    # rounding, ~100 eps_32 through transforms, end slopes and sweep
    return 2.2e-16 * 0.1 * N**4 * Ns**2 + 1e-13 if precision != "fp32" else 1e-5


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _case(Nx, Ny, N, Ns, seed):
    rng = np.random.default_rng(seed)
    g = (Nx, Ny) if Ny else (Nx,)
    f = rng.standard_normal((Ns,) + g + (N,))
    return f, rng.standard_normal(g), rng.standard_normal(g), rng


@pytest.mark.parametrize("bc", BCS)
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32_refine"])
def test_several_elements_forward_and_adjoint(cuda, shape, bc, precision):
    Nx, Ny, N, Ns = shape
    f, gl, gr, rng = _case(Nx, Ny, N, Ns, N + Ns)
    lam = 3.0
    if Ny:
        ref = O.solve3d(f, gl, gr, Lx=1.3, Ly=0.8, Lz=0.9, lam=lam, bc=bc)
        p = NonPeriodic3D(Nx, Ny, Ns * N, N, 0.0, 1.3, 0.0, 0.8, 0.0, 0.9, Lambda=lam, bc=bc, precision=precision)
    else:
        ref = O.solve2d(f, gl, gr, Lx=1.3, Ly=0.9, lam=lam, bc=bc)
        p = NonPeriodic2D(Nx, Ns * N, N, 0.0, 1.3, 0.0, 0.9, Lambda=lam, bc=bc, precision=precision)
    assert "multi_rows_kernel" in p.kernels()
    tol = _tol(N, Ns, precision)
    u = p.SolvePDE(_dev(f), _dev(gl), _dev(gr))
    assert rel_l2(u.cpu().numpy(), ref) < tol
    ubar = rng.standard_normal(f.shape)
    fbar, lbar, glb, grb = p.SolveAdjoint(_dev(ubar), u=_dev(ref), want_bc=True)
    fb, a, b = fbar.cpu().numpy(), glb.cpu().numpy(), grb.cpu().numpy()
    assert np.all(fb[..., 0] == 0) and np.all(fb[..., -1] == 0)
    lhs = float((ref * ubar).sum())
    rhs = float((f * fb).sum() + (gl * a).sum() + (gr * b).sum())
    # each side's rounding is relative to the products it sums
    scale = np.linalg.norm(ref) * np.linalg.norm(ubar) + np.linalg.norm(f) * np.linalg.norm(fb) \
        + np.linalg.norm(gl) * np.linalg.norm(a) + np.linalg.norm(gr) * np.linalg.norm(b)
    assert abs(lhs - rhs) < tol * scale
    want = float((fb * ref).sum())
    assert abs(lbar.item() - want) < tol * (np.linalg.norm(fb) * np.linalg.norm(ref) + 1e-300)


@pytest.mark.parametrize("shape", [s for s in SHAPES if not s[1]])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_several_elements_periodic(cuda, shape, precision):
    Nx, _, N, Ns = shape
    f, _, _, _ = _case(Nx, 0, N, Ns, N * Ns)
    ref = O.psolve2d(f, Lx=1.3, Ly=0.9, lam=3.0)
    p = Periodic2D(Nx, Ns * N, N, 0.0, 1.3, 0.0, 0.9, Lambda=3.0, precision=precision)
    u = p.SolvePDE(_dev(f)).cpu().numpy()
    assert rel_l2(u, ref) < _tol(N, Ns, precision)
