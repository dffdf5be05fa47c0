"""Planning a problem's tensor-core grid on the host: right, and cheap next to the
rest of a problem's creation also for k-sets that are refused (the structure
factor's: tens of thousands of runs of one row)."""

from __future__ import annotations

import importlib.util
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "xla-cco_b200" / "csrc"


def test_plans_are_right_and_cheap(tmp_path):
    spec = importlib.util.spec_from_file_location("cco_build", ROOT / "xla-cco_b200" / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    exe = tmp_path / "plan"
    # the library's host flags; what planning does not call stays unresolved
    cmd = [build.nvcc(), "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-Xcompiler", "-O2", "-Xcicc",
           "-O0", "-Xptxas", "-O0", "--expt-relaxed-constexpr", "-Xlinker", "--unresolved-symbols=ignore-all",
           f"-I{ROOT / 'include'}", f"-I{CSRC}", "-o", str(exe), str(ROOT / "tests" / "native" / "plan.cu")]  # fmt: skip
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    print(res.stdout)
    assert res.returncode == 0, res.stdout
