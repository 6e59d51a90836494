"""The plain FP32 form of the solver on batches beyond the 64 MB that its reconstruction GEMM writes at a time: the
images on both sides of a part's end, and the last one, against the same images in a solver of their own (another
order of the same FP32 sums: 2e-5 of V's norm, the bound the FP32 form is stated with)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openpv_gb300 import build
    build.build()
    return torch


@pytest.mark.parametrize("nb, ins, v1, nxp, per", [(400, (32, 32, 3), (16, 16, 64), 8, 341),
                                                   (300, (64, 64, 1), (16, 16, 64), 16, 256)])
def test_batch_in_parts(torch, nb, ins, v1, nxp, per):
    from openpv_gb300 import capi
    g = torch.Generator(device="cuda").manual_seed(nb)
    w = torch.randn((v1[2], nxp, nxp, ins[2]), device="cuda", generator=g)
    w /= w.square().sum(dim=(1, 2, 3), keepdim=True).sqrt()
    x = torch.randn((nb,) + ins, device="cuda", generator=g)
    v0 = 0.2 * torch.randn((nb,) + v1, device="cuda", generator=g)

    def solve(images):
        xs, vs = x[images].contiguous(), v0[images].contiguous()
        s = capi.LcaSolver(len(images), ins, v1, nxp, 0.1)
        s.set_weights(w)
        s.reset(vs)
        s.run(xs, 4, precision=capi.LCA_FP32)
        v, e = torch.empty_like(vs), torch.zeros(len(images), dtype=torch.float64, device="cuda")
        s.state(v)
        s.energy(xs, e)
        torch.cuda.synchronize()
        return v, e
    v, e = solve(list(range(nb)))
    some = [0, per - 1, per, nb - 1]
    vs, es = solve(some)
    for k, b in enumerate(some):
        assert (v[b] - vs[k]).norm() <= 2e-5 * vs[k].norm(), b
        assert abs(e[b] - es[k]) <= 1e-6 * abs(es[k]), b
