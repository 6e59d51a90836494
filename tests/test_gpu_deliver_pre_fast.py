"""The FAST presynaptic delivery kernels (deliver_pre_fast.cu) at the sizes where their tiles, column
slabs and entry chunks end, against the oracle.

Tolerance: both sides sum n = active entries reaching an output of products bounded by |a||w|, in FP32
but in different orders, so they differ by at most 2 n 2^-24 of the sum of the products' magnitudes;
that sum is taken from the oracle run on |a|, |w| and 0."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (pre nb, nx, ny, nf, halo), (post nx, ny, nf, halo), nxp, nyp, density, floats the weights start past a
# 256-byte boundary
CASES = [
    # wide post layers (24 features and more): columns
    ((1, 9, 5, 3, 1), (9, 5, 24, 0), 3, 3, 0.3, 0),        # three quarters of a warp, last column tile of one
    ((2, 8, 33, 2, 2), (8, 33, 25, 0), 5, 5, 0.2, 0),      # odd features: one per lane
    ((1, 17, 12, 5, 1), (17, 12, 72, 0), 3, 3, 0.2, 0),    # a partial slab
    ((1, 16, 16, 4, 0), (16, 16, 130, 0), 1, 1, 0.5, 0),   # two slabs, 1x1 patch
    ((1, 12, 10, 6, 2), (12, 10, 64, 0), 5, 5, 0.2, 1),    # weights not aligned for vector loads
    ((2, 24, 16, 7, 3), (6, 4, 40, 0), 2, 2, 0.2, 0),      # many-to-one x4, even patch
    ((1, 32, 20, 3, 9), (16, 10, 32, 0), 10, 10, 0.3, 0),  # window taller than the patch
    ((2, 6, 7, 5, 2), (24, 28, 32, 0), 16, 16, 0.3, 0),    # one-to-many x4, the tallest window
    ((1, 40, 36, 2, 8), (40, 36, 32, 0), 17, 17, 0.2, 0),  # taller than any window: shared-memory tiles
    # narrow post layers: shared-memory tiles
    ((1, 1, 1, 1, 0), (1, 1, 1, 0), 1, 1, 1.0, 0),
    ((3, 33, 31, 3, 1), (33, 31, 23, 0), 3, 3, 0.2, 0),
    ((2, 20, 20, 9, 5), (20, 20, 16, 0), 11, 11, 0.1, 0),  # patch of several lane blocks
    ((2, 10, 12, 40, 2), (40, 48, 1, 0), 16, 16, 0.1, 0),  # one-to-many x4
    ((1, 5, 3, 64, 3), (10, 6, 3, 1), 12, 8, 0.2, 0),      # patch larger than the layer, unequal axes
    ((4, 64, 48, 32, 2), (32, 24, 8, 0), 3, 3, 0.02, 0),   # many-to-one spikes
    ((1, 128, 96, 1, 1), (128, 96, 2, 0), 3, 3, 1.0, 0),   # dense image
    ((1, 70, 2, 3, 1), (70, 2, 5, 0), 3, 3, 0.0, 0),       # nothing active
    ((2, 16, 16, 60, 2), (32, 32, 3, 0), 8, 8, 0.1, 0),    # pairs of weights, patches starting off the vector grid
    ((2, 16, 16, 60, 2), (32, 32, 3, 0), 8, 8, 0.1, 1),    # the same with weights not aligned for vectors
    ((3, 9, 7, 6, 1), (9, 7, 8, 0), 3, 3, 0.3, 0),         # quads
    ((1, 12, 5, 200, 1), (48, 20, 2, 0), 8, 8, 0.2, 0),    # one-to-many x4 of two features: quads, one tile
    ((1, 16, 16, 300, 2), (64, 64, 1, 0), 16, 16, 0.1, 0),  # a tile of the whole image over a cluster
    ((2, 40, 44, 20, 4), (20, 22, 6, 0), 5, 5, 0.3, 0),    # pairs, many-to-one
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
def test_fast_presynaptic_delivery_at_tile_edges(cuda, oracle, case):
    torch = cuda
    from openpv_gb300 import capi
    (nb, nx, ny, nf, h), (qx, qy, qf, qh), nxp, nyp, p, skip = case
    rng = np.random.default_rng(nx * 31 + qf)
    pre, post = capi.Loc.make(nb, nx, ny, nf, h), capi.Loc.make(nb, qx, qy, qf, qh)
    opre, opost = oracle.Loc.make(nb, nx, ny, nf, h, h), oracle.Loc.make(nb, qx, qy, qf, qh, qh)
    a = ((rng.random(pre.ext_shape()) < p) * rng.normal(size=pre.ext_shape())).astype(np.float32)
    nk = max(1, nx // qx) * max(1, ny // qy) * nf
    w = rng.normal(0, 0.05, (nk, nyp, nxp, qf)).astype(np.float32)
    g0 = rng.normal(size=post.res_shape()).astype(np.float32)

    def reference(act, wgt, g):
        ent, num = oracle.compact(act.reshape(nb, -1))
        return oracle.deliver_pre(opre, opost, nxp, nyp, wgt, entries=ent, num_active=num, gsyn=g), ent, num

    ref, ent, num = reference(a, w, g0.copy())
    mag, _, _ = reference(np.abs(a), np.abs(w), np.abs(g0))
    n = max(1, int((a != 0).sum(axis=(1, 2, 3)).max()))
    tol = 2 * min(n, nf * nxp * nyp * max(1, nx // qx) * max(1, ny // qy) + 2) * 2.0 ** -24 * mag
    buf = torch.empty(w.size + skip, device="cuda")
    wd = buf[skip:]
    wd.copy_(torch.from_numpy(w.reshape(-1)))
    conn = capi.conn_desc(pre, post, nxp, nyp)
    outs = []
    for kw in ({"entries": torch.from_numpy(ent.view(np.uint8).copy()).cuda(), "num_active": torch.from_numpy(num).cuda()},
               {"a_ext": torch.from_numpy(a).cuda()}):
        for _ in range(2):
            g = torch.from_numpy(g0.copy()).cuda()
            capi.deliver_pre(conn, wd, g, **kw)
            outs.append(g.cpu().numpy())
        assert np.array_equal(outs[-1].view(np.uint32), outs[-2].view(np.uint32))  # the same order every time
        assert np.all(np.abs(outs[-1] - ref) <= tol), float(np.max(np.abs(outs[-1] - ref) / np.maximum(tol, 1e-30)))
