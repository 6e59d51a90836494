"""FAST presynaptic delivery from a layer four times as fine onto a wide one: the column kernel takes it at
every size.  Its sums are in SparseList order whatever the number of rows per block, so an image has the
same bits alone and in a batch that is large enough for the tallest blocks; and it is checked against the
oracle, with the bound of two orders of the same FP32 sum (2 n 2^-24 of the sum of magnitudes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openpv_gb300 import build
    build.build()
    return torch


@pytest.mark.parametrize("nb, n, nf, post_nf, nxp", [(8, 256, 1, 32, 3), (8, 256, 1, 24, 2), (6, 256, 1, 64, 3)])
def test_many_to_one_by_four_batch_equals_images(cuda, oracle, nb, n, nf, post_nf, nxp):
    torch = cuda
    from openpv_gb300 import capi
    h = 4 * nxp
    g = torch.Generator(device="cuda").manual_seed(n + post_nf)

    def deliver(a, w):
        k = a.shape[0]
        pre, post = capi.Loc.make(k, 4 * n, 4 * n, nf, h), capi.Loc.make(k, n, n, post_nf, 0)
        e = torch.empty(k, pre.num_ext, dtype=torch.int64, device="cuda")
        num = torch.zeros(k, dtype=torch.int64, device="cuda")
        capi.compact_active(a, k, pre.num_ext, e, num)
        out = torch.zeros(post.res_shape(), device="cuda")
        capi.deliver_pre(capi.conn_desc(pre, post, nxp, nxp), w, out, entries=e, num_active=num)
        return out, e, num

    a = torch.randn((nb, 4 * n + 2 * h, 4 * n + 2 * h, nf), device="cuda", generator=g)
    a *= torch.rand(a.shape, device="cuda", generator=g) < 0.02
    w = torch.randn((16 * nf, nxp, nxp, post_nf), device="cuda", generator=g) * 0.05
    out, _, _ = deliver(a, w)
    for b in range(nb):
        one, e, num = deliver(a[b:b + 1].contiguous(), w)
        assert torch.equal(out[b].view(torch.int32), one[0].view(torch.int32)), b
    opre, opost = oracle.Loc.make(1, 4 * n, 4 * n, nf, h, h), oracle.Loc.make(1, n, n, post_nf, 0, 0)
    ref, mag = (oracle.deliver_pre(opre, opost, nxp, nxp, f(w.cpu().numpy()), entries=ent, num_active=cnt,
                                   gsyn=np.zeros((1, n, n, post_nf), np.float32))
                for f in (lambda v: v, np.abs)
                for ent, cnt in [oracle.compact(f(a[-1].cpu().numpy()).reshape(1, -1))])
    k = 16 * nf * nxp * nxp
    assert np.all(np.abs(one.cpu().numpy() - ref) <= 2 * (k + 1) * 2.0 ** -24 * mag)
