"""The FP32 postsynaptic delivery at the sizes where its tiles, K steps and cluster divisions end,
against the oracle in FP64.

Tolerance: K products summed in FP32 in any order, added to GSyn: at most (K + 2) 2^-24 times the sum of
the magnitudes, which the FP64 oracle gives for |a|, |w| and |GSyn|."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (pre nb, nx, ny, nf, halo), (post nx, ny, nf, halo), nxp, nyp
CASES = [
    ((1, 1, 1, 1, 0), (1, 1, 1, 0), 1, 1),            # K = 1
    ((1, 5, 3, 7, 1), (5, 3, 5, 0), 3, 3),            # one ragged tile
    ((1, 16, 16, 64, 3), (16, 16, 64, 0), 7, 7),      # few positions, long K: divided over a cluster
    ((1, 12, 11, 33, 2), (12, 11, 65, 1), 5, 5),      # odd K, one feature beyond a tile
    ((1, 64, 64, 1, 6), (16, 16, 130, 2), 4, 4),      # stride 4, 130 features
    ((2, 64, 64, 8, 1), (64, 64, 129, 0), 3, 3),      # 128 x 128 tiles with a remainder
    ((9, 48, 40, 16, 2), (24, 20, 64, 0), 3, 3),      # even stride, rows of 96 values
    ((1, 16, 20, 40, 8), (64, 80, 3, 0), 16, 16),     # one-to-many x4, three features: narrow tile
    ((2, 20, 12, 9, 8), (40, 24, 12, 0), 10, 10),     # one-to-many x2, twelve features
    ((3, 130, 70, 3, 1), (130, 70, 1, 0), 3, 3),      # one feature
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
def test_post_delivery_at_tile_edges(cuda, oracle, case):
    torch = cuda
    from openpv_gb300 import capi
    (nb, nx, ny, nf, h), (qx, qy, qf, qh), nxp, nyp = case
    rng = np.random.default_rng(nx + 7 * qf)
    pre, post = capi.Loc.make(nb, nx, ny, nf, h), capi.Loc.make(nb, qx, qy, qf, qh)
    opre, opost = oracle.Loc.make(nb, nx, ny, nf, h, h), oracle.Loc.make(nb, qx, qy, qf, qh, qh)
    px, py = oracle.post_patch_size(nxp, nx, qx), oracle.post_patch_size(nyp, ny, qy)
    kernels = max(1, qx // nx) * max(1, qy // ny) * qf
    a = rng.normal(size=pre.ext_shape()).astype(np.float32)
    w = rng.normal(0, 0.05, (kernels, py, px, nf)).astype(np.float32)
    g0 = rng.normal(size=post.res_shape()).astype(np.float32)
    d = lambda x: x.astype(np.float64)  # noqa: E731
    ref = d(g0) + oracle.deliver_post_f64(opre, opost, px, py, d(w), d(a))
    mag = d(np.abs(g0)) + oracle.deliver_post_f64(opre, opost, px, py, d(np.abs(w)), d(np.abs(a)))
    T = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    outs = []
    for _ in range(2):
        g = T(g0.copy())
        capi.deliver_post(capi.conn_desc(pre, post, nxp, nyp), T(a), T(w), g)
        outs.append(g.cpu().numpy())
    assert np.array_equal(outs[0].view(np.uint32), outs[1].view(np.uint32))
    tol = (px * py * nf + 2) * 2.0 ** -24 * mag
    assert np.all(np.abs(outs[0] - ref) <= tol), float(np.max(np.abs(outs[0] - ref) / tol))
