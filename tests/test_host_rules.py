"""Host-side rules of the kernel dispatch, checked as compiled code without a
GPU (tests/cpp): which addresses a launch's descriptors let its kernels touch."""
import re
import subprocess
from pathlib import Path

import pytest

from t1m_gb300 import build

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("name", ["store_flags", "piece_loads", "stream_splits", "skinny_blocks",
                                  "pieces_pay", "stream_pays", "small_form"])
def test_host_rule(built_lib, name):
    out = ROOT / "tests" / "_build" / name
    out.parent.mkdir(parents=True, exist_ok=True)
    cmd = [build.nvcc(), "-std=c++17", "-O1", f"-I{build.CSRC}", f"-I{build.INCLUDE}",
           str(ROOT / "tests" / "cpp" / f"{name}.cpp"), f"-L{build.OUT_DIR}", "-lt1m_cuda",
           "-Xlinker", f"-rpath={build.OUT_DIR}", "-o", str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(out)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def _kernels():
    """(name, body lines) of every kernel of the library."""
    for src in sorted(build.CSRC.glob("*.cu")):
        lines = src.read_text().splitlines()
        for i, line in enumerate(lines):
            if "__global__" not in line:
                continue
            head = " ".join(lines[i:i + 3])
            name = re.search(r"(\w+)\(const|(\w+)\(const __grid_constant__", head.split("__global__")[1]
                             .replace("__launch_bounds__", ""))
            end = next(j for j in range(i, len(lines)) if lines[j] == "}")
            yield name.group(1) if name else head, [x.strip() for x in lines[i:end]]


def test_dependent_kernels_order_their_reads():
    """A kernel that may start before the ones ahead of it have ended waits for
    them, in every thread, before it lets others start and before it reads
    what they wrote.  A split pass that runs beside another orders its reads by
    a fence instead (begin_split) and waits at its end."""
    text = "\n".join(p.read_text() for p in build.CSRC.glob("*.cu"))
    dependent = {n for call in re.findall(r"launch_dependent\(([^;]*)", text)
                 for n in re.findall(r"\b(\w+)<", call.split("dim3")[0])} - {"static_cast"}
    bodies = dict(_kernels())
    assert {"split_pieces", "split_pieces_step", "splitk_reduce"} <= dependent
    for name in dependent | {"tc1m_pieces"}:
        body = bodies[name]
        first = next(x for x in body if re.search("begin_|release_dependents|__ldg", x))
        if name.startswith("split_pieces"):
            assert first.startswith("begin_split("), (name, first)
            assert body[-1].endswith("beside) begin_dependent();"), (name, body[-1])
        else:
            assert first == "begin_dependent();", (name, first)
    begin = text[text.index("void begin_split("):]
    assert re.sub(r"\s+", " ", begin[:begin.index("\n}")]) == (
        "void begin_split(bool beside) { if (beside) __threadfence(); else begin_dependent(); "
        "release_dependents();")
