"""Complex passes of length 512 on 512-thread CTAs: their time beside that of a copy
of the same bytes."""
import pytest
import torch

from mpi_b200 import Helmholtz3DFD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,precision", [((1024, 512, 64), "fp32"), ((256, 512, 128), "fp64")])
def test_complex_passes_near_the_copy_rate(cuda, shape, precision):
    Nx, Ny, N = shape
    p = Helmholtz3DFD(Nx, Ny, N, 0.0, 1.0, 0.0, 1.0, 0.0, 1.0, Lambda=20.0, precision=precision)
    p.set_launch_variants([8] * 4, 0)
    f = torch.randn(Nx, Ny, N, dtype=torch.float64, device=cuda)
    out = torch.empty_like(f)
    p.SolvePDE(f, out=out)
    p.enable_stage_timing(True)
    passes = []
    for _ in range(12):
        p.SolvePDE(f, out=out)
        t = p.stage_times()
        passes.append(min(t["fft_y"], t["ifft_y"]))
    # the spectrum once in and once out
    a = torch.randn((Nx // 2 + 1) * Ny * N * (2 if precision == "fp64" else 1), dtype=torch.float64, device=cuda)
    b = torch.empty_like(a)
    copies = []
    for _ in range(12):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        b.copy_(a)
        e1.record()
        e1.synchronize()
        copies.append(e0.elapsed_time(e1))
    # 1.25 copies; with the warps that spare registers cost, 1.5 (FP32) and 1.8 (FP64)
    assert min(passes) < 1.4 * min(copies)
