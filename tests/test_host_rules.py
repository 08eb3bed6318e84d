"""Host-side rules of the kernel dispatch, checked as compiled code without a
GPU (tests/cpp): which addresses a launch's descriptors let its kernels touch."""
import subprocess
from pathlib import Path

import pytest

from t1m_gb300 import build

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("name", ["store_flags", "piece_loads"])
def test_host_rule(name):
    out = ROOT / "tests" / "_build" / name
    out.parent.mkdir(parents=True, exist_ok=True)
    cmd = [build.nvcc(), "-std=c++17", "-O1", f"-I{build.CSRC}", f"-I{build.INCLUDE}",
           str(ROOT / "tests" / "cpp" / f"{name}.cpp"), "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
