"""The gradient of unrolled LCA at sizes where the split-plane GEMMs' tiles, chunks and splits of positions
end, on the library-GEMM path (patches whose size is not a multiple of eight), and with segments of one
step, of more steps than there are and with a short last one; against the gradient in float64 by
autograd.  dW within 1e-4 of max|dW| and the loss within 1e-5, the bounds the gradient is stated with."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# nb, image (y, x, c), v1 (y, x, f), patch, steps, checkpoint every
CASES = [
    (1, (32, 32, 1), (8, 8, 8), 16, 7, 3),        # 64 positions, eight features
    (3, (32, 32, 1), (16, 16, 40), 8, 5, 10),     # columns beyond a 32-run, a segment longer than the run
    (2, (32, 32, 3), (16, 16, 136), 8, 4, 1),     # two feature tiles, the second of eight; every step a segment
    (5, (64, 64, 1), (16, 16, 200), 16, 6, 2),
    (1, (12, 20, 1), (6, 10, 72), 4, 5, 2),       # 60 positions: a chunk of positions that ends early
    (2, (20, 12, 2), (10, 6, 24), 6, 5, 2),       # patches of 72 values, generic geometry
    (2, (16, 16, 1), (8, 8, 24), 6, 4, 2),        # patches of 36 values: library GEMMs
    (1, (16, 16, 1), (8, 8, 20), 8, 4, 2),        # 20 features: library GEMMs
    (40, (64, 64, 1), (16, 16, 128), 16, 3, 2),   # more rows than one wave of tiles
]


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from openpv_gb300 import build
    build.build()
    return torch


def reference(torch, w, x, v1, P, steps, vt, lam):
    F = torch.nn.functional
    nb, n, S = x.shape[0], x.shape[1:3], x.shape[1] // v1[0]
    kw = dict(kernel_size=P, stride=S, padding=(P - S) // 2)
    wd = w.double().requires_grad_(True)
    m = wd.permute(0, 3, 1, 2).reshape(w.shape[0], -1)
    xc = x.double().permute(0, 3, 1, 2)
    recon = lambda a: F.fold((a @ m).transpose(1, 2), tuple(n), **kw)  # noqa: E731
    soft = lambda v: torch.where(v >= vt, v - vt, torch.zeros_like(v))  # noqa: E731
    e = float(np.float32(math.exp(-1.0 / 100.0)))
    v = torch.zeros((nb, v1[0] * v1[1], v1[2]), dtype=torch.float64, device="cuda")
    for _ in range(steps):
        a = soft(v)
        v = e * v + (1 - e) * (F.unfold(xc - recon(a), **kw).transpose(1, 2) @ m.T + a)
    a = soft(v)
    loss = 0.5 * (xc - recon(a)).square().sum() + lam * a.abs().sum()
    loss.backward()
    return wd.grad, loss.item()


@pytest.mark.parametrize("case", CASES)
def test_gradient_at_tile_edges(torch, case):
    from openpv_gb300 import capi
    nb, ins, v1, P, steps, every = case
    g = torch.Generator(device="cuda").manual_seed(nb + P)
    w = torch.randn((v1[2], P, P, ins[2]), device="cuda", generator=g)
    w /= w.square().sum(dim=(1, 2, 3), keepdim=True).sqrt()
    x = 20.0 * torch.randn((nb,) + ins, device="cuda", generator=g)  # drives V over the threshold within a few steps
    vt = float(np.float32(0.1))
    h = capi.LcaGrad(nb, ins, v1, P, 0.1, 0.1, steps, checkpoint_every=every)
    dw, loss = torch.empty_like(w), torch.zeros(1, dtype=torch.float64, device="cuda")
    outs = []
    for _ in range(2):
        dw.fill_(float("nan"))
        h.run(w, x, dw, loss)
        torch.cuda.synchronize()
        outs.append(dw.clone())
    assert torch.equal(outs[0].view(torch.int32), outs[1].view(torch.int32))
    ref, lref = reference(torch, w, x, v1, P, steps, vt, vt)
    assert abs(loss.item() - lref) <= 1e-5 * abs(lref)
    assert (outs[0].double() - ref).abs().max() <= 1e-4 * ref.abs().max()
