"""Kernels that need more than the default dynamic shared memory are opted in on
every device a process uses, not on the first one only. Runs the host code of the
launches against a runtime with two devices made of plain C++ (no GPU)."""

from __future__ import annotations

import importlib.util
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "xla-cco_b200" / "csrc"


def _nvcc() -> str:
    spec = importlib.util.spec_from_file_location("cco_build", ROOT / "xla-cco_b200" / "build.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod.nvcc()


def test_launches_with_large_shared_memory_on_a_second_device(tmp_path):
    flags = ["-gencode", "arch=compute_100a,code=sm_100a", "-Xcicc", "-O0", "-Xptxas", "-O0", "-std=c++17",
             "--expt-relaxed-constexpr", "-cudart", "none", f"-I{ROOT / 'include'}", f"-I{CSRC}"]  # fmt: skip
    native = ROOT / "tests" / "native"
    srcs = [native / "two_devices.cu", native / "two_devices_runtime.cpp", CSRC / "cco_hessian.cu",
            CSRC / "cco_persist.cu"]  # fmt: skip
    objs = [tmp_path / (s.name + ".o") for s in srcs]
    jobs = [subprocess.Popen([_nvcc(), *flags, "-c", "-o", str(o), str(s)], stdout=subprocess.PIPE,
                             stderr=subprocess.STDOUT, text=True) for s, o in zip(srcs, objs)]  # fmt: skip
    for j in jobs:
        out, _ = j.communicate()
        assert j.returncode == 0, out
    exe = tmp_path / "two_devices"
    res = subprocess.run(["g++", "-o", str(exe), *map(str, objs)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout


def test_no_attribute_is_set_once_per_process():
    """Every opt-in runs per device (OncePerDevice) or per call."""
    for f in sorted(CSRC.glob("*.cu*")):
        text = f.read_text()
        assert "call_once" not in text and "once_flag" not in text, f.name
        assert not re.search(r"static\s+(const\s+)?(bool|cudaError_t)\s+\w+\s*=", text), f.name
