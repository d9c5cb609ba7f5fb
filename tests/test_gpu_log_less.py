"""The score's acceptance test (log_less, csrc/crmathf.cuh) decides with a
single-precision logarithm where that one cannot be wrong: over all 2^32 words its
verdict is the double logarithm's at bounds on both sides of log u, at the line
between the two (1e-4) and far from it, and the single-precision logarithm is
within the 1e-5 that the line relies on."""
import os
import subprocess

import pytest

pytest.importorskip("torch")
from conftest import require_cuda  # noqa: E402
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_log_less_equals_the_double_logarithm(tmp_path):
    require_cuda()
    exe = str(tmp_path / "log_less_test")
    r = subprocess.run([os.path.join(CUDA, "bin", "nvcc"), "-gencode", "arch=compute_100a,code=sm_100a", "-O3",
                        "-std=c++17", f"-I{ROOT}/mckl_b200/csrc", os.path.join(ROOT, "tests", "cpp", "log_less_test.cu"),
                        "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    wrong, worst = out.stdout.split()
    assert int(wrong) == 0 and float(worst) <= 1e-5, out.stdout
