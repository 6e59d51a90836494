"""The forms that index with 64 bits, at the smallest sizes that take them: the Hebbian update on post activities of
more than 2^31 values, and the row walk on layers of more than 2^31 neurons (17 GB on the device); and the FAST
presynaptic delivery of a patch that neither FAST kernel takes."""
import pytest

from tests import test_gpu_deliver_pre_fast as fast

pytestmark = pytest.mark.gpu
cuda = fast.cuda


@pytest.fixture()
def torch(cuda):
    if cuda.cuda.mem_get_info()[0] < 30 << 30:
        pytest.skip("needs 30 GB of free device memory")
    yield cuda
    cuda.cuda.empty_cache()


def test_hebbian_64bit_offsets(torch):
    """Two images whose post activity exceeds 2^31 values in all, four active neurons; the same float products and
    sums in the same order, by torch."""
    from openpv_gb300 import capi
    nb, n, f = 2, 64, 262145
    pre, post = capi.Loc.make(nb, n, n, 1, 0), capi.Loc.make(nb, n, n, f, 0)
    assert nb * post.num_ext > 1 << 31
    a = torch.zeros(pre.ext_shape(), device="cuda")
    r = torch.zeros(post.ext_shape(), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    want = torch.zeros(f, device="cuda")
    for k, (b, y, x) in enumerate([(0, 0, 0), (0, 63, 62), (1, 0, 1), (1, 63, 63)]):
        a[b, y, x, 0] = 0.3 + k
        r[b, y, x] = torch.randn(f, device="cuda", generator=g)
        want = want + (0.7 * a[b, y, x, 0]) * r[b, y, x]
    dw = torch.full((f,), float("nan"), device="cuda")
    capi.hebbian_dw(capi.conn_desc(pre, post, 1, 1), 0.7, a, r, dw)
    assert torch.equal(dw.view(torch.int32), want.view(torch.int32))


def test_row_walk_64bit_units(torch):
    from openpv_gb300 import capi
    nx, ny = 65537, 32769
    L = capi.Loc.make(1, nx, ny, 1, 1)
    assert L.num_res > (1 << 31) - 1 and nx % 4
    v = torch.empty((ny, nx), device="cuda")
    g = torch.Generator(device="cuda").manual_seed(2)
    rows = [0, 1, 16383, 16384, 32767, 32768]
    v.fill_(0.5)
    for y in rows:
        v[y] = torch.randn(nx, device="cuda", generator=g)
    a = torch.full((ny + 2, nx + 2), -7.0, device="cuda")
    vt = 0.25
    capi.ann_activity(L, v, vt, 0.0, float("inf"), vt, 0.0, a)
    for y in rows:
        want = torch.where(v[y] < vt, torch.zeros_like(v[y]), v[y] - vt)
        assert torch.equal(a[y + 1, 1:-1], want), y
    assert (a[[0, -1]] == -7.0).all() and (a[:, 0] == -7.0).all() and (a[:, -1] == -7.0).all()
    for y0 in range(2, ny - 1, 4096):  # the rows in between
        y1 = min(y0 + 4096, ny - 1)
        skip = [y - y0 for y in rows if y0 <= y < y1]
        ok = (a[y0 + 1:y1 + 1, 1:-1] == 0.25).all(dim=1)
        ok[skip] = True
        assert ok.all(), y0


@pytest.mark.parametrize("case", [((1, 64, 64, 2, 0), (4, 4, 3, 0), 61, 61, 0.02, 0),
                                  ((2, 48, 32, 3, 4), (3, 2, 30, 0), 41, 90, 0.1, 0)])
def test_patch_beyond_both_fast_kernels(cuda, oracle, case):
    """Sixteen times as fine, 61x61: too many rows for the columns' table, too large for a shared-memory tile."""
    fast.test_fast_presynaptic_delivery_at_tile_edges(cuda, oracle, case)
