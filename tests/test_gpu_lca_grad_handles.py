"""Several gradient handles alive at once: none may depend on another's sizes.  Against the gradient in
float64 by autograd, dW within 1e-4 of max|dW| and the loss within 1e-5."""
import numpy as np
import pytest

from tests.test_gpu_lca_grad_sizes import reference

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openpv_gb300 import build
    build.build()
    return torch


def make(torch, nb, ins, v1, P, steps, every):
    from openpv_gb300 import capi
    g = torch.Generator(device="cuda").manual_seed(P)
    w = torch.randn((v1[2], P, P, ins[2]), device="cuda", generator=g)
    w /= w.square().sum(dim=(1, 2, 3), keepdim=True).sqrt()
    x = 20.0 * torch.randn((nb,) + ins, device="cuda", generator=g)
    return capi.LcaGrad(nb, ins, v1, P, 0.1, 0.1, steps, checkpoint_every=every), w, x, steps


def check(torch, h, w, x, steps, v1, P):
    vt = float(np.float32(0.1))
    dw, loss = torch.full_like(w, float("nan")), torch.zeros(1, dtype=torch.float64, device="cuda")
    h.run(w, x, dw, loss)
    torch.cuda.synchronize()
    ref, lref = reference(torch, w, x, v1, P, steps, vt, vt)
    assert abs(loss.item() - lref) <= 1e-5 * abs(lref)
    assert (dw.double() - ref).abs().max() <= 1e-4 * ref.abs().max()


@pytest.mark.parametrize("wide, small", [
    # patch windows of 90 KB and of 2 KB in the kernel for any geometry
    ((1, (16, 128, 8), (4, 32, 8), 16), (1, (16, 16, 2), (8, 8, 8), 6)),
    # 78 KB and 3 KB in the kernel for 8x8 patches of colour images at stride 2
    ((1, (16, 640, 3), (8, 320, 16), 8), (1, (16, 16, 3), (8, 8, 16), 8)),
])
def test_smaller_handle_made_later(torch, wide, small):
    first = make(torch, *wide, 3, 2)
    second = make(torch, *small, 3, 2)
    check(torch, *first, wide[2], wide[3])
    check(torch, *second, small[2], small[3])
    check(torch, *first, wide[2], wide[3])  # and once more
