"""The dot product's scratch (its counter must be zero before the first call)
when the allocation or the clear is refused: tests/cpp/dot_scratch_driver.cpp."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_refused_clear_leaves_no_scratch(tmp_path):
    from sep_code_gb300 import build
    inc = Path(build._nvcc()).parent.parent / "include"
    if shutil.which("g++") is None or not inc.is_dir():
        pytest.skip("no g++ or CUDA headers")
    exe = tmp_path / "driver"
    subprocess.run(["g++", "-std=c++17", "-Wall", f"-I{build.CSRC}", f"-I{inc}",
                    str(ROOT / "tests/cpp/dot_scratch_driver.cpp"), "-o", str(exe)], check=True, capture_output=True,
                   text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
