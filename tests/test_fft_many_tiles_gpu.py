"""Complex passes on 512-thread CTAs: the kernel for many tiles begins beyond two waves
of the other one; solves just below and just above that line, last tiles partly
filled, against the same solve on 256-thread CTAs."""
import pytest
import torch

from mpi_b200 import Helmholtz3DFD
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu

# (Nx, Ny, N) -> (Nx / 2 + 1) N / 8 tiles: 591 and 593 about 4 x 148 (FP32 length 512, two CTAs an
# SM), 296 and 297 about 2 x 148 (one CTA an SM: FP64 length 512, FP32 length 1024)
CASES = [((32, 512, 278), "fp32"), ((32, 512, 279), "fp32"), ((8, 512, 473), "fp64"), ((8, 512, 475), "fp64"),
         ((8, 1024, 473), "fp32"), ((8, 1024, 475), "fp32")]


@pytest.mark.parametrize("shape,precision", CASES)
def test_many_tiles(cuda, shape, precision):
    Nx, Ny, N = shape
    p = Helmholtz3DFD(Nx, Ny, N, 0.0, 1.0, 0.0, 1.0, 0.0, 1.0, Lambda=20.0, precision=precision)
    f = torch.randn(Nx, Ny, N, dtype=torch.float64, device=cuda)
    got = []
    for v in (0, 8):
        p.set_launch_variants([0, v, v, 0], 0)
        got.append(p.SolvePDE(f).cpu().numpy())
    # two transforms and their inverses round by log2(L) eps each: 40 eps, of white right-hand sides
    assert rel_l2(got[1], got[0]) < (100 * 2.2e-16 if precision == "fp64" else 100 * 1.2e-7)
