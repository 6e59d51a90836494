"""Host threads that call one entry point at the same time, on streams of their own, with sizes that run the
same kernel with different amounts of shared memory: every call goes through, with the bits that one thread
alone gets."""
import threading
import time

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


def hebbian(torch, capi, seed, post_nf):
    """3x3 patches of 4 features: 8 warps (64 KB of lists) for 18 weights, 16 (128 KB) for 504."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    pre, post = capi.Loc.make(1, 12, 10, 4, 1), capi.Loc.make(1, 12, 10, post_nf, 0)
    a = torch.randn(pre.ext_shape(), device="cuda", generator=g)
    r = torch.randn(post.ext_shape(), device="cuda", generator=g)
    conn = capi.conn_desc(pre, post, 3, 3)

    def make():
        dw = torch.empty(4 * 9 * post_nf, device="cuda")
        return lambda stream: capi.hebbian_dw(conn, 0.5, a, r, dw, stream=stream), dw
    return make


def scatter(torch, capi, seed, nb, n, nf):
    """5x5 patches of 12 features: tiles of 62 KB for the small layer, of 112 KB for the large one."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    pre, post = capi.Loc.make(nb, n, n, nf, 2), capi.Loc.make(nb, n, n, 12, 0)
    a = torch.randn(pre.ext_shape(), device="cuda", generator=g)
    a *= torch.rand(pre.ext_shape(), device="cuda", generator=g) < 0.01
    e = torch.empty(nb, pre.num_ext, dtype=torch.int64, device="cuda")
    num = torch.zeros(nb, dtype=torch.int64, device="cuda")
    capi.compact_active(a, nb, pre.num_ext, e, num)
    w = torch.randn(nf * 25 * 12, device="cuda", generator=g)
    conn = capi.conn_desc(pre, post, 5, 5)

    def make():
        gs = torch.empty(post.res_shape(), device="cuda")

        def call(stream):
            gs.zero_()
            capi.deliver_pre(conn, w, gs, entries=e, num_active=num, stream=stream)
        return call, gs
    return make


def gemm(torch, capi, seed, entry, n):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn((128, 256), device="cuda", generator=g).bfloat16()
    b = torch.randn((256, n) if entry == "tc_gemm_bf16_kn" else (n, 256), device="cuda", generator=g).bfloat16()

    def make():
        c, err = torch.empty((128, n), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
        return lambda stream: getattr(capi, entry)(a, b, c, 128, n, 256, err, stream=stream), c
    return make


GEMMS = ["tc_gemm_bf16", "tc_gemm_bf16_kn", "tc_gemm_bf16_atmem"]


@pytest.mark.parametrize("kernel", ["hebbian", "scatter"] + GEMMS)
def test_same_kernel_from_several_threads(torch, kernel):
    from openpv_gb300 import capi
    calls = {"hebbian": lambda: [hebbian(torch, capi, 1, 56), hebbian(torch, capi, 2, 2)],
             "scatter": lambda: [scatter(torch, capi, 1, 4, 64, 64), scatter(torch, capi, 2, 2, 32, 16)],
             **{e: lambda e=e: [gemm(torch, capi, 1, e, 256), gemm(torch, capi, 2, e, 128)] for e in GEMMS}}[kernel]()
    alone = []
    for c in calls:
        call, out = c()
        call(torch.cuda.current_stream())
        alone.append(out.cpu().numpy())
    errors, wrong, stop = [], [], time.monotonic() + 3.0

    def work(i):
        s = torch.cuda.Stream()
        try:
            with torch.cuda.stream(s):
                call, out = calls[i]()
                while time.monotonic() < stop and not errors:
                    for _ in range(200):
                        call(s)
                    s.synchronize()
                    if not np.array_equal(out.cpu().numpy().view(np.uint32), alone[i].view(np.uint32)):
                        wrong.append(i)
        except Exception as e:  # noqa: BLE001
            errors.append(f"thread of size {i}: {e}")

    threads = [threading.Thread(target=work, args=(i % 2,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors and not wrong, (errors, wrong)


def test_solvers_made_while_another_runs(torch):
    """One thread makes solvers of small images while another captures and runs one of large images, which takes
    more shared memory in the same kernels."""
    from openpv_gb300 import capi
    w = torch.randn((64, 8, 8, 1), device="cuda")
    w /= w.square().sum(dim=(1, 2, 3), keepdim=True).sqrt()
    xs = [torch.randn((2, 64, 64, 1), device="cuda") for _ in range(2)]
    big = capi.LcaSolver(2, (64, 64, 1), (32, 32, 64), 8, 0.1)
    big.set_weights(w)
    torch.cuda.synchronize()
    errors, stop = [], time.monotonic() + 3.0

    def run():
        s = torch.cuda.Stream()
        try:
            k = 0
            while time.monotonic() < stop and not errors:
                big.reset(stream=s)
                big.run(xs[k & 1], 6, 2, precision=capi.LCA_BF16, stream=s)  # another input: captured again
                k += 1
                s.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(f"run: {e}")

    def make():
        try:
            while time.monotonic() < stop and not errors:
                capi.LcaSolver(1, (32, 32, 1), (16, 16, 64), 8, 0.1).close()
        except Exception as e:  # noqa: BLE001
            errors.append(f"make: {e}")

    threads = [threading.Thread(target=run), threading.Thread(target=make)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors and big.error_flag() == 0, errors
