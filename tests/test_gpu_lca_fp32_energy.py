"""The energy probe after FP32 timesteps subtracts the last step's reconstruction from the image that it is given,
which need not be the one the steps ran on (an input buffer refilled for the next display period); against the
same in float64 from the solver's own states.  The BF16 form's probe keeps the residual of its run."""
import numpy as np
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


@pytest.mark.parametrize("nb, ins, v1, nxp", [(3, (32, 32, 1), (16, 16, 64), 8), (2, (32, 32, 3), (16, 16, 128), 8),
                                              (2, (64, 64, 1), (16, 16, 64), 16)])
def test_energy_of_another_image(torch, nb, ins, v1, nxp):
    from openpv_gb300 import capi
    g = torch.Generator(device="cuda").manual_seed(nxp)
    w = torch.randn((v1[2], nxp, nxp, ins[2]), device="cuda", generator=g)
    w /= w.square().sum(dim=(1, 2, 3), keepdim=True).sqrt()
    x, other = (torch.randn((nb,) + ins, device="cuda", generator=g) for _ in range(2))
    v0 = 0.2 * torch.randn((nb,) + v1, device="cuda", generator=g)
    s = capi.LcaSolver(nb, ins, v1, nxp, 0.1)
    s.set_weights(w)
    s.reset(v0)
    before, after = torch.empty_like(v0), torch.empty_like(v0)
    s.run(x, 2, precision=capi.LCA_FP32)
    s.state(a=before)
    s.run(x, 1, precision=capi.LCA_FP32)
    s.state(a=after)
    S = ins[0] // v1[0]
    m = w.double().permute(0, 3, 1, 2).reshape(v1[2], -1)
    rec = torch.nn.functional.fold((before.double().reshape(nb, -1, v1[2]) @ m).transpose(1, 2), ins[:2], kernel_size=nxp,
                                   stride=S, padding=(nxp - S) // 2).permute(0, 2, 3, 1)
    cost = float(np.float32(0.1)) * after.double().abs().sum(dim=(1, 2, 3))
    e = torch.zeros(nb, dtype=torch.float64, device="cuda")
    for image in (x, other):
        s.energy(image, e)
        torch.cuda.synchronize()
        want = 0.5 * (image.double() - rec).square().sum(dim=(1, 2, 3)) + cost
        assert ((e - want).abs() <= 1e-5 * want).all(), (e, want)
    s.reset(v0)  # no step yet: the image itself
    s.energy(other, e)
    torch.cuda.synchronize()
    want = 0.5 * other.double().square().sum(dim=(1, 2, 3)) + \
        float(np.float32(0.1)) * torch.where(v0 >= np.float32(0.1), v0 - np.float32(0.1), 0.0).double().sum(dim=(1, 2, 3))
    assert ((e - want).abs() <= 1e-5 * want).all()
