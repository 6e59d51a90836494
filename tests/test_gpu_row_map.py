"""The layer updates at the row shapes that decide their vector width and at sizes where a block of
units ends or spans several batch elements: bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nb, nx, ny, nf, halo (x), halo (y)
LOCS = [
    (1, 1, 128, 8, 0, 0),    # rows of 8 values
    (3, 5, 37, 3, 1, 2),     # nothing divides by four
    (2, 8, 16, 4, 3, 0),     # rows and halo in fours
    (2, 6, 40, 6, 1, 1),     # rows in fours, halo not
    (9, 7, 21, 1, 2, 2),     # 147 neurons: a block spans 14 batch elements
    (1, 33, 31, 2, 0, 1),
    (5, 16, 16, 32, 2, 2),
]


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openpv_gb300 import build
    build.build()
    return torch


@pytest.mark.parametrize("shape", LOCS)
@pytest.mark.parametrize("skip", [0, 1])
def test_updates_over_row_shapes(cuda, oracle, shape, skip):
    """skip: floats that every buffer starts past an aligned address."""
    torch = cuda
    from openpv_gb300 import capi
    nb, nx, ny, nf, mx, my = shape
    loc, oloc = capi.Loc.make(nb, nx, ny, nf, mx, my), oracle.Loc.make(nb, nx, ny, nf, mx, my)
    rng = np.random.default_rng(nx + 100 * nf)
    f32 = lambda s: rng.normal(size=s).astype(np.float32)  # noqa: E731
    gsyn, v0, a0, drive = f32((2,) + loc.res_shape()), f32(loc.res_shape()), f32(loc.ext_shape()), f32(loc.res_shape())
    dt = rng.uniform(0.5, 2.0, nb)

    def T(x):
        x = np.ascontiguousarray(x)
        buf = torch.empty(x.size + skip, device="cuda")
        buf[skip:] = torch.from_numpy(x.reshape(-1)).cuda()
        return buf[skip:]

    H = lambda t, like: t.cpu().numpy().reshape(like.shape).view(np.uint32)  # noqa: E731
    same = lambda t, ref: np.testing.assert_array_equal(H(t, ref), ref.view(np.uint32))  # noqa: E731
    dtd = torch.from_numpy(dt).cuda()
    g_ref = oracle.gsyn_accumulate(gsyn, [1.0, -0.5])
    g = T(np.zeros_like(g_ref))
    capi.gsyn_accumulate(g_ref.size, [1.0, -0.5], T(gsyn), g)
    same(g, g_ref)
    v_ref = oracle.lca_update(oloc, g_ref, a0, v0, dt, 100.0)
    v, a = T(v0), T(a0)
    capi.lca_update(loc, True, dtd, 100.0, g, a, v)
    same(v, v_ref)
    a_ref = oracle.ann_activity(oloc, v_ref, 0.1, 0.0, 1.0, 0.05, 0.3, a_ext=a0)
    capi.ann_activity(loc, v, 0.1, 0.0, 1.0, 0.05, 0.3, a)
    same(a, a_ref)
    # the fused form leaves the same state
    desc = capi.LcaLayerDesc(loc, 2, (1.0, -0.5, 0.0, 0.0), 1, 100.0, 0.1, 0.0, 1.0, 0.05, 0.3)
    v2, a2 = T(v0), T(a0)
    capi.lca_layer_update(desc, T(gsyn), dtd, v2, a2)
    same(v2, v_ref)
    same(a2, a_ref)
    vm, d = T(v0), T(drive)
    vm_ref, d_ref = oracle.momentum_lca_update(oloc, g_ref, a0, drive, v0, dt, 100.0, 0.3)
    capi.momentum_lca_update(loc, True, 0.3, dtd, 100.0, g, T(a0), d, vm)
    same(vm, vm_ref)
    same(d, d_ref)
    vi = T(v0)
    capi.ista_update(loc, 0.1, dtd, 100.0, g, T(a0), vi)
    same(vi, oracle.ista_update(oloc, g_ref, a0, v0, dt, 100.0, 0.1))
