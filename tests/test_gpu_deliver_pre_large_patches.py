"""FAST presynaptic delivery of patches taller than the column kernel's window of 16 rows (passes of equal
heights) and of large patches onto narrow layers, at the sizes where the passes and the choice of the kernel
change; checked as the other FAST cases are."""
import pytest

from tests import test_gpu_deliver_pre_fast as fast

pytestmark = pytest.mark.gpu
cuda = fast.cuda

CASES = [
    # columns in passes
    ((2, 24, 24, 3, 8), (24, 24, 130, 0), 5, 17, 0.1, 0),     # eight and nine rows, two slabs of features
    ((2, 64, 64, 3, 16), (64, 64, 25, 0), 7, 33, 0.05, 0),    # three of eleven, one feature a lane
    ((1, 24, 24, 8, 16), (24, 24, 130, 0), 7, 33, 0.1, 0),    # (the dense form of it too)
    ((1, 24, 24, 8, 16), (24, 24, 130, 0), 7, 33, 0.1, 1),    # weights not aligned for vectors
    ((2, 20, 30, 5, 2), (80, 120, 40, 0), 4, 20, 0.2, 0),     # one-to-many x4
    ((2, 160, 160, 2, 18), (40, 40, 130, 0), 3, 19, 0.05, 0),  # many-to-one x4
    ((8, 512, 512, 2, 8), (32, 32, 24, 0), 1, 25, 0.02, 0),   # many-to-one x16: the second pass has too many rows
    # narrow layers
    ((2, 40, 44, 17, 12), (40, 44, 21, 0), 25, 23, 0.05, 0),  # a tile would be mostly margin: columns
    ((3, 8, 60, 7, 6), (8, 60, 21, 0), 13, 27, 0.1, 0),
    # small layers, which the scatter kernel takes
    ((2, 20, 33, 3, 2), (20, 33, 24, 0), 3, 17, 0.2, 0),
    ((1, 4, 3, 2, 5), (4, 3, 30, 0), 3, 35, 0.5, 0),
    ((2, 6, 7, 3, 4), (6, 7, 5, 0), 23, 21, 0.3, 0),
]


@pytest.mark.parametrize("case", CASES)
def test_large_patches(cuda, oracle, case):
    fast.test_fast_presynaptic_delivery_at_tile_edges(cuda, oracle, case)
