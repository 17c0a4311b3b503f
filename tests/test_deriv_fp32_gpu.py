"""GLL derivative of FP32 arrays: computed in FP64 and rounded once, on the packed
kernel (16-byte aligned arrays, tails of one to three values) and on the general one
(arrays that start off alignment)."""
import numpy as np
import pytest
import torch

from mpi_b200 import NonPeriodic2D, NonPeriodic3D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,N,Ns", [((4,), 3, 1), ((4,), 5, 3), ((8, 4), 16, 1), ((4, 4), 33, 2), ((64, 4), 65, 1),
                                       ((4, 4), 129, 1), ((16, 16), 7, 1)])
@pytest.mark.parametrize("shift", [0, 1])
def test_fp32_gll_derivative(cuda, dims, N, Ns, shift):
    rng = np.random.default_rng(N)
    if len(dims) == 1:
        plan = NonPeriodic2D(dims[0], N * Ns, N, 0.0, 1.0, 0.0, 2.0, Lambda=1.0, precision="fp32")
        first, second = plan.FirstDerivativeY, plan.SecondDerivativeY
    else:
        plan = NonPeriodic3D(*dims, N * Ns, N, 0.0, 1.0, 0.0, 1.0, 0.0, 2.0, Lambda=1.0, precision="fp32")
        first, second = plan.FirstDerivativeZ, plan.SecondDerivativeZ
    plan.set_io_bytes(4)
    _, D, D2 = plan.grid()
    n = Ns * int(np.prod(dims)) * N
    buf = torch.empty(n + shift, dtype=torch.float32, device="cuda")
    u = buf[shift:].view(Ns, *dims, N)
    u.copy_(torch.from_numpy(rng.standard_normal(tuple(u.shape))))
    for fn, M in ((first, D), (second, D2)):
        want = u.double().cpu() @ M.T
        size = u.double().abs().cpu() @ M.abs().T  # what the FP64 sums may lose
        out = torch.full((n + shift,), float("nan"), dtype=torch.float32, device="cuda")[shift:].view(u.shape)
        got = fn(u, out=out).double().cpu()
        assert ((got - want).abs() <= 2.0 ** -24 * want.abs() + 1e-13 * size + 1e-37).all()
        same = u.clone()
        if shift == 0:
            fn(same, out=same)  # in place
            assert torch.equal(same.double().cpu(), got)
