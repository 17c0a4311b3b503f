"""Creation of plans with several GLL elements: the interface factors of all shifts
cost little beside the rest of the plan."""
import time

import pytest
import torch

from mpi_b200 import NonPeriodic3D

pytestmark = pytest.mark.gpu


def test_creation_time_hardly_depends_on_the_elements(cuda):
    def create(Ns):
        torch.cuda.synchronize()
        t = time.perf_counter()
        p = NonPeriodic3D(256, 256, 6 * Ns, 6, 0.0, 1.0, 0.0, 1.0, 0.0, 1.0, Lambda=1.0, bc=(1.0, 0.5, 0.7, 2.0))
        torch.cuda.synchronize()
        t = time.perf_counter() - t
        p.DestroyPDEPlan()
        return t

    for Ns in (2, 60):
        create(Ns)  # launch variants are measured once per shape
    few, many = [], []
    # 16641 shifts; 1.05 measured, factors worked out on the host 1.54.  The fastest of each
    # counts; a busy host gets more tries
    for _ in range(100):
        few.append(create(2))
        many.append(create(60))
        if len(many) >= 8 and min(many) < 1.25 * min(few):
            break
    assert min(many) < 1.25 * min(few)
