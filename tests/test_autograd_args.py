"""Arguments of the evolve autograd function that the forward refuses (no GPU needed: the
checks come before any CUDA call)."""
import pytest

torch = pytest.importorskip("torch")

import ridgedetection_b200 as rdb  # noqa: E402
from ridgedetection_b200 import autograd as adj  # noqa: E402


def test_negative_checkpoint_interval_is_refused_by_the_forward():
    P = torch.zeros((4, 2))
    with pytest.raises(rdb.RDError, match="iteration counts"):
        adj.evolve_function().apply(P, torch.tensor([0]), 0.1, 1, -1)


@pytest.mark.parametrize("shape", [(8,), (2, 2, 2)])
def test_points_are_a_matrix(shape):
    with pytest.raises(ValueError):
        adj.evolve_means_device(torch.zeros(shape), torch.zeros((1, 2)), 0.1, 1)
