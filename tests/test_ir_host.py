"""Host build of the IR reader (csrc/ir.cuh): operands of malformed IR."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_ir_operands_stay_inside(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "ir_test"
    subprocess.run([cxx, "-O1", "-std=c++17", "-fsanitize=undefined",
                    "-fno-sanitize-recover=all", "-I", str(ROOT / "15418-project_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp_host" / "ir_test.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("OK"), out.stdout + out.stderr
