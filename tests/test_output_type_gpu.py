"""SolvePDE returns a plain tensor whatever class of tensor f is."""
import pytest
import torch

from mpi_b200 import NonPeriodic2D

pytestmark = pytest.mark.gpu


class Field(torch.Tensor):
    pass


@pytest.mark.parametrize("wrap", [lambda t: t, lambda t: t.as_subclass(Field), torch.nn.Parameter])
def test_solution_is_a_plain_tensor(cuda, wrap):
    p = NonPeriodic2D(8, 9, 9, 0.0, 1.0, 0.0, 1.0, Lambda=1.0)
    f = torch.randn(8, 9, dtype=torch.float64, device=cuda)
    u = p.SolvePDE(wrap(f))
    assert type(u) is torch.Tensor and not u.requires_grad
    assert torch.equal(u, p.SolvePDE(f))
