"""The gradient of layers with fewer neurons than the library path's probe GEMM spans (512), and of one position
or one feature; against the gradient in float64 by autograd, as the other sizes."""
import pytest

from tests import test_gpu_lca_grad_sizes as sizes

pytestmark = pytest.mark.gpu
torch = sizes.torch

CASES = [
    (1, (4, 4, 1), (1, 1, 1), 4, 3, 1),
    (2, (12, 4, 3), (3, 1, 2), 12, 5, 7),
    (3, (16, 6, 3), (8, 3, 3), 6, 3, 5),
    (1, (3, 15, 1), (3, 15, 9), 3, 4, 2),     # stride 1
    (1, (8, 8, 1), (2, 2, 8), 8, 4, 2),       # the split-plane path: one tile, mostly beyond the matrix
    (1, (2, 2, 2), (1, 1, 16), 4, 2, 1),
]


@pytest.mark.parametrize("case", CASES)
def test_gradient_of_tiny_layers(torch, case):
    sizes.test_gradient_at_tile_edges(torch, case)
