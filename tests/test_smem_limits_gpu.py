"""Plans of different sizes share kernels: the shared memory that one of them asks for
does not take away another's, neither by being created later nor from another
thread."""
import math
import threading

import pytest
import torch

from mpi_b200 import BatchNonPeriodic2D, NonPeriodic2D

pytestmark = pytest.mark.gpu

TWO_PI = 2.0 * math.pi


def test_small_batch_created_after_a_large_one(cuda):
    def batch(Nx, N):
        b = BatchNonPeriodic2D([Nx] * 3, [N] * 3, [1.0, 2.0, 3.0], 0.0, TWO_PI, -1.0, 1.0)
        b.set_graph(False)
        return b, torch.randn(b.total, dtype=torch.float64, device=cuda)

    large, f = batch(512, 129)
    want = large.solve(f)
    small, g = batch(8, 5)
    small.solve(g)
    assert torch.equal(large.solve(f), want)


def test_threads_with_plans_of_two_sizes(cuda):
    # 52 KB and 77 KB a CTA in the same kernel; four threads of each size
    sizes = [(40, 60), (100, 30)] * 4
    plans = [NonPeriodic2D(4, Ns * N, N, 0.0, TWO_PI, -1.0, 1.0, Lambda=1.0) for N, Ns in sizes]
    fields = [torch.randn(Ns, 4, N, dtype=torch.float64, device=cuda) for N, Ns in sizes]
    want = [p.SolvePDE(f) for p, f in zip(plans, fields)]
    outs = [torch.empty_like(f) for f in fields]
    streams = [torch.cuda.Stream() for _ in sizes]
    torch.cuda.synchronize()
    start, errors = threading.Barrier(len(sizes)), []

    def work(p, f, out, s):
        solve, args = p._lib.helm_solve, (p._plan, f.data_ptr(), None, None, out.data_ptr(), s.cuda_stream)
        start.wait()
        for _ in range(3000):
            st = solve(*args)
            if st:
                errors.append(st)
                return

    threads = [threading.Thread(target=work, args=a) for a in zip(plans, fields, outs, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for out, w in zip(outs, want):
        assert torch.equal(out, w)
