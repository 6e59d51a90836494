"""The gradient's windows where a row of positions is divided over several blocks (few bands, large patches of a
geometry without a kernel of its own): parts of equal and unequal sizes, several bands, a part that ends the row."""
import pytest

from tests import test_gpu_lca_grad_sizes as sizes

pytestmark = pytest.mark.gpu
torch = sizes.torch

CASES = [
    (3, (56, 76, 3), (14, 19, 8), 16, 4, 3),      # parts of four positions, the last of three
    (1, (24, 200, 1), (6, 50, 16), 12, 3, 2),     # two positions a part
    (2, (20, 66, 4), (10, 33, 8), 14, 3, 1),      # an odd row
    (1, (5, 23, 8), (5, 23, 8), 9, 3, 2),         # stride 1
    (40, (16, 16, 3), (4, 4, 8), 16, 3, 2),       # enough bands: whole rows
]


@pytest.mark.parametrize("case", CASES)
def test_gradient_with_divided_rows(torch, case):
    sizes.test_gradient_at_tile_edges(torch, case)
