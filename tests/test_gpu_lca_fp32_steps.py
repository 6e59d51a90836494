"""The plain FP32 form's three kernels over feature counts and batches that leave partial GEMM tiles, and
a threshold with width and ceiling, against the oracle; 12 timesteps, V within 1e-5 of max|V| and the
L1 energy within 1e-5, the form's stated bounds."""
import numpy as np
import pytest

from tests.test_gpu_lca_solver import dictionary, one_over_f, torch  # noqa: F401

pytestmark = pytest.mark.gpu

# nb, (in y, x, c), (v1 y, x, f), patch, VWidth, AMax
CASES = [
    (1, (32, 32, 1), (16, 16, 64), 8, 0.0, np.inf),
    (5, (32, 32, 3), (16, 16, 192), 8, 0.05, 0.6),
    (3, (64, 64, 1), (16, 16, 320), 16, 0.0, np.inf),
    (2, (16, 128, 3), (8, 64, 64), 8, 0.0, np.inf),  # wide: two rows of positions per 128
]


@pytest.mark.parametrize("case", CASES)
def test_fp32_steps_match_oracle(torch, oracle, case):  # noqa: F811
    from openpv_gb300 import capi
    nb, ins, v1s, P, width, amax = case
    rng = np.random.default_rng(v1s[2] + nb)
    w, x = dictionary(rng, v1s[2], P, ins[2]), one_over_f(rng, nb, *ins)
    v0 = rng.normal(0, 0.15, (nb,) + v1s).astype(np.float32)
    # the solver's timestep from the oracle's pieces (its first step reconstructs the initial activity)
    v1 = oracle.Loc.make(nb, v1s[1], v1s[0], v1s[2], oracle.required_margin(v1s[1], ins[1], P),
                         oracle.required_margin(v1s[0], ins[0], P))
    q = P * v1s[1] // ins[1]
    er = oracle.Loc.make(nb, ins[1], ins[0], ins[2], oracle.required_margin(ins[1], v1s[1], q),
                         oracle.required_margin(ins[0], v1s[0], q))
    threshold = lambda v: oracle.ann_activity(v1, v, 0.1, 0.0, amax, 0.1, width)  # noqa: E731
    v_ref, a_ref, dt = v0, threshold(v0), np.ones(nb)
    for _ in range(12):
        err = x - oracle.deliver_pre(v1, er, P, P, w, a_ext=a_ref)
        err_ext = np.zeros(er.ext_shape(), np.float32)
        h = er.halo
        err_ext[:, h.up:h.up + ins[0], h.lt:h.lt + ins[1], :] = err
        v_ref = oracle.lca_update(v1, oracle.deliver_post(er, v1, P, P, w, err_ext), a_ref, v_ref, dt, 100.0)
        a_ref = threshold(v_ref)
    e_ref = 0.5 * (err.astype(np.float64) ** 2).sum(axis=(1, 2, 3)) + float(np.float32(0.1)) * np.abs(
        a_ref.astype(np.float64)).sum(axis=(1, 2, 3))
    s = capi.LcaSolver(nb, ins, v1s, P, 0.1, AMax=float(amax), VWidth=width)
    s.set_weights(torch.from_numpy(w).cuda())
    s.reset(torch.from_numpy(v0).cuda())
    xd = torch.from_numpy(x).cuda()
    s.run(xd, 12, precision=capi.LCA_FP32)
    v, e = torch.zeros((nb,) + v1s, device="cuda"), torch.zeros(nb, dtype=torch.float64, device="cuda")
    s.state(v, None)
    assert np.abs(v.cpu().numpy() - v_ref).max() <= 1e-5 * np.abs(v_ref).max()
    s.energy(xd, e)
    np.testing.assert_allclose(e.cpu().numpy(), e_ref, rtol=1e-5)
