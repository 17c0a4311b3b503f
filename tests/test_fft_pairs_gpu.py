"""The FFT passes move two neighbouring real columns (or their two spectrum
values) as one access where the addresses allow it.  Arrays that start half a
pair off, odd row strides and odd column counts take the separate accesses; both
have to give the same solve, adjoint and derivatives."""
import numpy as np
import pytest
import torch

from mpi_b200 import Helmholtz3DFD, NonPeriodic2D, NonPeriodic3D

pytestmark = pytest.mark.gpu

ROBIN = (1.0, 0.5, 0.7, 2.0)


def _at(a, shift, dtype):
    """A contiguous CUDA copy of `a` that starts `shift` elements into its storage."""
    buf = torch.empty(a.size + shift, dtype=dtype, device="cuda")
    t = buf[shift:].view(a.shape)
    t.copy_(torch.from_numpy(a))
    return t


def _close(a, b, eps):
    # the same operations on the same values: at most a few contractions of a*b+c differ
    a, b = a.double(), b.double()
    assert (a - b).abs().max().item() <= 64 * eps * b.abs().max().item()


@pytest.mark.parametrize("dims,N", [((8,), 9), ((64,), 10), ((1024,), 6), ((4, 4), 5), ((16, 8), 9), ((256, 4), 8),
                                    ((512, 4), 7), ((32, 128), 6)])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32_io4"])
def test_pairs_and_single_columns_agree(cuda, dims, N, precision):
    rng = np.random.default_rng(sum(dims) + N)
    prec, io = precision[:4], torch.float32 if precision == "fp32_io4" else torch.float64
    kw = dict(Lambda=1.5, bc=ROBIN, precision=prec)
    # two elements in 2D, so that odd N has batches half a pair off
    if len(dims) == 1:
        plan, shape = NonPeriodic2D(dims[0], 2 * N, N, 0.0, 1.3, 0.0, 0.9, **kw), (2, dims[0], N)
    else:
        plan, shape = NonPeriodic3D(*dims, N, N, 0.0, 1.3, 0.0, 0.7, 0.0, 0.9, **kw), (1, *dims, N)
    if io == torch.float32:
        plan.set_io_bytes(4)
    eps = 2.2e-16 if prec == "fp64" else 6e-8
    f, obs = rng.standard_normal(shape), rng.standard_normal(shape)
    gl, gr = (torch.from_numpy(rng.standard_normal(dims)).cuda() for _ in range(2))
    got = []
    for shift in (0, 1):
        fs = _at(f, shift, io)
        u = plan.SolvePDE(fs, gl, gr, out=_at(f, shift, io))
        res = [u, plan.FirstDerivativeX(fs, out=_at(f, shift, io)), plan.SecondDerivativeX(fs, out=_at(f, shift, io))]
        if io == torch.float64:
            res += [t for t in plan.SolveAdjointMisfit(u, _at(obs, shift, io), want_bc=True)]
        got.append([t.clone() for t in res])
    # the misfit gradient starts from this solve's own u, one solve's rounding off
    for a, b in zip(got[1], got[0]):
        _close(a, b, eps)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32_refine"])
@pytest.mark.parametrize("shape", [(4, 4, 3), (16, 8, 12), (256, 4, 9), (1024, 4, 6)])
def test_fd_pairs_and_single_columns_agree(cuda, precision, shape):
    rng = np.random.default_rng(sum(shape))
    plan = Helmholtz3DFD(*shape, 0.0, 1.0, 0.0, 2.0, 0.0, 1.5, Lambda=30.0, bc=ROBIN, precision=precision)
    f, obs = rng.standard_normal(shape), rng.standard_normal(shape)
    gl, gr = (torch.from_numpy(rng.standard_normal(shape[:2])).cuda() for _ in range(2))
    eps = 6e-8 if precision == "fp32" else 2.2e-16 if precision == "fp64" else 1e-13
    got = []
    for shift in (0, 1):
        u = plan.SolvePDE(_at(f, shift, torch.float64), gl, gr, out=_at(f, shift, torch.float64))
        res = [u, *plan.SolveAdjointMisfit(u, _at(obs, shift, torch.float64), want_bc=True)]
        got.append([t.clone() for t in res])
    for a, b in zip(got[1], got[0]):
        _close(a, b, eps)
