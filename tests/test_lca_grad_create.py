"""pvgpu_lca_grad_create on the host, with counted allocations and a stand-in for cuBLAS
(tests/grad_create): what it hands to cuBLAS lies inside its buffers at the smallest sizes, and destroy gives
everything back."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "grad_create")
ROOT = os.path.dirname(os.path.dirname(HERE))
OK, OOM = 0, 2


@pytest.fixture(scope="module")
def create(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("grad_create")
    exe, so = str(d / "harness"), str(d / "libfakecublas.so")
    subprocess.check_call(["g++", "-shared", "-fPIC", "-o", so, os.path.join(HERE, "fake_cublas.cpp")])
    # device code is not run: ptxas need not optimise it
    subprocess.check_call([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-Xptxas", "-O0", "-std=c++17", "-w",
                           "--expt-relaxed-constexpr", "-Xcompiler", "-rdynamic", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(ROOT, "openpv_gb300", "csrc"), "-o", exe, os.path.join(HERE, "harness.cu"),
                           "-ldl"])

    def run(*lines):
        r = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, timeout=60,
                           env=dict(os.environ, PVGPU_CUBLAS=so))
        assert r.returncode == 0, r.stderr
        out = [ln.split() for ln in r.stdout.splitlines()]
        assert len(out) == len(lines)
        return [(int(s), int(b), float(p), int(left), int(tc)) for s, b, p, left, tc in out]
    return run


def line(nb, ins, v1, nxp, steps, every, budget_mb=1e6, vthresh=0.1):
    (iy, ix, c), (vy, vx, f) = ins, v1
    return f"{budget_mb} {nb} {ix} {iy} {c} {vx} {vy} {f} {nxp} {vthresh} {steps} {every}"


def test_library_path_probe_stays_in_its_buffer(create):
    """The probe GEMM's operands span 512 floats; a layer may have fewer neurons."""
    cases = [line(1, (4, 4, 1), (1, 1, 1), 4, 1, 1), line(1, (4, 12, 3), (1, 3, 2), 12, 10, 7),
             line(3, (16, 6, 3), (8, 3, 3), 6, 3, 5), line(1, (4, 4, 1), (2, 2, 8), 4, 2, 1, vthresh=-0.1),
             line(2, (64, 64, 1), (16, 16, 20), 16, 4, 2)]
    for got in create(*cases):
        assert got[:2] == (OK, 0) and got[3:] == (0, 0), got


def test_library_path_where_the_split_plane_one_does_not_fit(create):
    """100 steps with a checkpoint before each: 2.7 GB on the split-plane path, 1.9 on the other."""
    case = lambda mb: line(8, (32, 32, 1), (16, 16, 2048), 8, 100, 1, budget_mb=mb)  # noqa: E731
    roomy, tight, short = create(case(3000), case(2300), case(1500))
    assert roomy[:2] == (OK, 0) and roomy[3:] == (0, 1) and roomy[2] > 2300
    assert tight[:2] == (OK, 0) and tight[3:] == (0, 0) and tight[2] <= 2300
    assert short[:2] == (OOM, 0) and short[3] == 0
