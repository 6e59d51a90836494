"""The Hebbian update where the patch is wider or taller than the post layer, so that a warp first picks the
entries that put a weight of its own inside: bit for bit against the oracle, over the feature groups and weights
per lane that the launch chooses from."""
import pytest

from tests import test_gpu_hebbian_lists as lists

pytestmark = pytest.mark.gpu
cuda = lists.cuda

CASES = [
    ((1, 1, 1, 1, 0), (1, 1, 1, 0), 3, 1, 1.0),
    ((4, 10, 2, 22, 13), (10, 2, 2, 0), 15, 21, 0.7),     # one feature a CTA, one weight a lane, 32 warps
    ((1, 4, 1, 107, 1), (4, 1, 60, 0), 7, 13, 0.95),      # eight weights a lane
    ((2, 2, 4, 111, 5), (2, 4, 7, 3), 17, 11, 0.9),   # two weights a lane
    ((3, 3, 2, 300, 3), (3, 2, 12, 0), 5, 7, 0.5),        # two features a CTA
    ((2, 3, 4, 600, 3), (3, 4, 9, 1), 5, 5, 0.3),         # four
    ((1, 3, 4, 1100, 3), (3, 4, 6, 2), 5, 7, 0.05),       # eight
    ((1, 3, 4, 1100, 3), (3, 4, 90, 0), 5, 7, 0.4),       # eight, eight weights a lane
    ((6, 2, 4, 3, 10), (2, 4, 80, 0), 17, 13, 0.6),       # more than 32 entries a list and segment
    ((2, 12, 2, 5, 6), (3, 2, 20, 1), 4, 5, 0.6),         # many-to-one across
    ((2, 4, 1, 6, 4), (16, 4, 7, 0), 20, 8, 0.6),         # one-to-many
    ((1, 6, 5, 9, 0), (6, 5, 40, 0), 13, 11, 0.0),        # nothing active
]


@pytest.mark.parametrize("case", CASES)
def test_patch_exceeds_layer(cuda, oracle, case):
    lists.test_hebbian_lists_bitexact(cuda, oracle, case)
