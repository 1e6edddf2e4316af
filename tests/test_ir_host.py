"""Host builds of the IR reader (csrc/ir.cuh): operands of malformed IR, and what
a launch provides for an IR."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def _run_host_test(tmp_path, name):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / name
    subprocess.run([cxx, "-O1", "-std=c++17", "-fsanitize=undefined",
                    "-fno-sanitize-recover=all", "-I", str(ROOT / "15418-project_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp_host" / f"{name}.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr


def test_ir_operands_stay_inside(tmp_path):
    _run_host_test(tmp_path, "ir_test")


def test_launch_needs_of_an_ir(tmp_path):
    _run_host_test(tmp_path, "ir_needs_test")
