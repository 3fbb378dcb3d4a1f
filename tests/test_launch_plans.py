"""CPU: the host-side launch plans, compiled without optimisation and with the host compiler's undefined-behaviour checks
(tests/sanitize/*_plans.cu), over calls and devices of many sizes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("what", ["launch", "attention", "strip"])
def test_plans_under_ubsan(what, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc) or shutil.which("g++") is None:
        pytest.skip("no compiler")
    exe = str(tmp_path / "plans")
    san = ["-fsanitize=undefined", "-fno-sanitize-recover=undefined"]
    cmd = [nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O0", "-w", "--expt-relaxed-constexpr", *[a for f in san for a in ("-Xcompiler", f)],
           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "lmdeploy_b200", "csrc"), os.path.join(ROOT, "tests", "sanitize", what + "_plans.cu"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0 and "cannot find" in r.stderr and "ubsan" in r.stderr:
        pytest.skip("sanitizer runtime not installed")
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "plans ok" in r.stdout
