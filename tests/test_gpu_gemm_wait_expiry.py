"""The bounded waits of the gradient's GEMMs, run out on purpose on operands that never arrive, without a fault or a
hang: the error word is set and nothing written, the next kernel of the run ends at once, and the context and tensor
memory stay usable."""
import pytest

from tests import test_gpu_lca_grad_sizes as sizes

pytestmark = pytest.mark.gpu
torch = sizes.torch
LIMIT = 200_000_000  # ns, that of every bounded wait


@pytest.mark.parametrize("chunks", [1, 2, 5])  # fewer stages than the ring has, and more (the load lane gives up too)
def test_gemm_waits_expire(torch, chunks):
    from openpv_gb300 import capi
    st, word, first, second, wrote = capi.selftest_gemm_expiry(chunks)
    assert st == capi.PVGPU_ERR_TIMEOUT and word == 1 and wrote == 0
    # one limit for the waits, one for each copy that would be in flight (at most three)
    assert LIMIT <= first <= (1 + min(chunks, 3)) * LIMIT + LIMIT // 2, first
    assert second < LIMIT // 4, second
    sizes.test_gradient_at_tile_edges(torch, (2, (32, 32, 3), (16, 16, 136), 8, 4, 1))


def test_arguments_and_error_flag(torch):
    from openpv_gb300 import capi
    for chunks in (0, -1, 65):
        assert capi.selftest_gemm_expiry(chunks)[0] == capi.PVGPU_ERR_BAD_ARG
    for f in (24, 20):  # split-plane and library GEMMs
        h = capi.LcaGrad(1, (16, 16, 1), (8, 8, f), 8, 0.1, 0.1, 3)
        assert h.error_flag() == 0
        w, x = torch.randn((f, 8, 8, 1), device="cuda"), torch.randn((1, 16, 16, 1), device="cuda")
        dw, loss = torch.empty_like(w), torch.zeros(1, dtype=torch.float64, device="cuda")
        h.run(w, x, dw, loss)
        torch.cuda.synchronize()
        assert h.error_flag() == 0 and torch.isfinite(dw).all()
