"""A state array is used in place only where one page-locked allocation or registration holds all of it: an
array that begins in one and ends in another has ordinary memory between."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
TOP = 2 ** 64


def test_one_range_holds_the_whole_array(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "pinned_range_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(ROOT / "physics-engine_gb300" / "csrc"), "-I", "/usr/local/cuda/include",
                    str(ROOT / "tests" / "pinned_range_check.cpp"), "-o", str(exe)], check=True, capture_output=True)
    cases = [((65536, 4096, 65536, 4096), 1), ((65536, 4096, 65540, 4092), 1), ((65536, 4096, 65540, 4093), 0), ((65536, 4096, 65535, 8), 0),
             ((65536, 4096, 69632, 1), 0), ((65536, 4096, 69631, 1), 1), ((65536, 4096, 66000, 131072), 0),   # ends in a range further on
             ((TOP - 4096, 4096, TOP - 8, 8), 1), ((TOP - 4096, 4096, TOP - 8, 9), 0), ((4096, TOP - 4096, 8192, TOP - 8192), 1),
             ((65536, 0, 65536, 4), 0), ((0, 0, 65536, 4), 0)]
    out = subprocess.run([str(exe)], input="".join("%d %d %d %d\n" % c for c, _ in cases), check=True, capture_output=True, text=True).stdout.split()
    assert [int(x) for x in out] == [w for _, w in cases]
