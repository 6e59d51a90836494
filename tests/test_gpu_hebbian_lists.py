"""The Hebbian kernel's per-feature lists at the sizes where its loads, segments, feature groups and
weight slabs end: bit for bit against the oracle, whose summation order it keeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (pre nb, nx, ny, nf, halo), (post nx, ny, nf, halo), nxp, nyp, density
CASES = [
    ((1, 1, 1, 1, 0), (1, 1, 1, 0), 1, 1, 1.0),
    ((2, 33, 9, 1, 1), (33, 9, 2, 1), 3, 3, 1.0),       # one feature, dense: full lists, several segments
    ((2, 70, 40, 3, 2), (70, 40, 1, 0), 5, 5, 0.4),     # three features, rows of a partial load
    ((1, 12, 10, 300, 1), (12, 10, 5, 2), 3, 3, 0.1),   # features not a multiple of the group
    ((2, 16, 16, 1100, 2), (32, 32, 1, 3), 8, 8, 0.05),  # eight features a CTA
    ((1, 9, 8, 6, 2), (9, 8, 40, 2), 5, 5, 0.3),        # 1000 weights: slabs beyond one CTA's warps
    ((1, 9, 7, 9, 3), (9, 7, 64, 3), 7, 7, 0.3),        # 3136 weights
    ((2, 32, 16, 5, 6), (8, 4, 3, 2), 4, 4, 0.3),       # many-to-one x4: sixteen kernel phases
    ((1, 8, 6, 20, 5), (32, 24, 2, 1), 16, 16, 0.2),    # one-to-many x4, halo wider than the patch needs
    ((2, 20, 12, 7, 0), (20, 12, 3, 0), 7, 7, 0.0),     # nothing active
    ((2, 9, 7, 1, 3), (9, 7, 130, 3), 9, 9, 0.5),       # 10530 weights, one feature: eleven CTAs of 32 warps
    ((1, 6, 5, 100, 2), (6, 5, 44, 2), 5, 5, 0.3),      # 1100 weights, a hundred features: two weights a lane
    ((1, 6, 5, 100, 2), (6, 5, 90, 1), 5, 5, 0.3),      # 2250: eight a lane
    ((1, 7, 6, 300, 2), (7, 6, 20, 0), 5, 5, 0.2),      # two features a CTA, 500 weights
    ((1, 7, 6, 600, 2), (7, 6, 11, 0), 5, 5, 0.2),      # four features a CTA, 275 weights: two a lane
    ((1, 7, 6, 1100, 2), (7, 6, 4, 2), 5, 5, 0.2),      # eight features a CTA, 100 weights
    ((1, 7, 6, 1100, 2), (7, 6, 8, 2), 5, 5, 0.2),      # 200: two a lane
    ((1, 7, 6, 1100, 2), (7, 6, 24, 2), 5, 5, 0.2),     # 600: eight a lane
]


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openpv_gb300 import build
    build.build()
    return torch


@pytest.mark.parametrize("case", CASES)
def test_hebbian_lists_bitexact(cuda, oracle, case):
    torch = cuda
    from openpv_gb300 import capi
    (nb, nx, ny, nf, h), (qx, qy, qf, qh), nxp, nyp, p = case
    rng = np.random.default_rng(nx * 13 + nf)
    pre, post = capi.Loc.make(nb, nx, ny, nf, h), capi.Loc.make(nb, qx, qy, qf, qh)
    a = ((rng.random(pre.ext_shape()) < p) * rng.normal(size=pre.ext_shape())).astype(np.float32)
    r = rng.normal(size=post.ext_shape()).astype(np.float32)
    ref = oracle.hebbian_dw(oracle.Loc.make(nb, nx, ny, nf, h, h), oracle.Loc.make(nb, qx, qy, qf, qh, qh), nxp, nyp, a,
                            r, 0.7)
    dw = torch.full((ref.size,), np.nan, device="cuda")
    capi.hebbian_dw(capi.conn_desc(pre, post, nxp, nyp), 0.7, torch.from_numpy(a).cuda(), torch.from_numpy(r).cuda(), dw)
    assert np.array_equal(dw.cpu().numpy().reshape(ref.shape).view(np.uint32), ref.view(np.uint32))


def test_hebbian_inactive_neurons_skip_nonfinite_post(cuda, oracle):
    """Zeros are skipped, not multiplied: an infinite post value under inactive neurons only leaves
    every weight finite."""
    torch = cuda
    from openpv_gb300 import capi
    pre, post = capi.Loc.make(1, 12, 12, 4, 1), capi.Loc.make(1, 12, 12, 2, 0)
    a = np.zeros(pre.ext_shape(), np.float32)
    a[0, 3, 3, 1] = 2.0
    r = np.full(post.ext_shape(), np.inf, np.float32)
    r[0, 1:4, 1:4] = 0.5  # all that the active neuron's 3x3 patch reaches
    dw = torch.full((4 * 9 * 2,), np.nan, device="cuda")
    capi.hebbian_dw(capi.conn_desc(pre, post, 3, 3), 1.0, torch.from_numpy(a).cuda(), torch.from_numpy(r).cuda(), dw)
    got = dw.cpu().numpy().reshape(4, 9, 2)
    assert np.all(got[1] == 1.0) and np.all(got[[0, 2, 3]] == 0.0)
