"""The bounded wait of the dedispersion pipelines (gaffa_b200/csrc/mbarrier.cuh):
when it runs out it says so to the whole warp and in the status word."""
import subprocess
from pathlib import Path

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]


def test_a_wait_that_runs_out_answers_for_the_warp(tmp_path):
    from gaffa_b200 import build
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    exe = tmp_path / "wait_warp_check"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, str(ROOT / "tests" / "wait_warp_check.cu"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr
