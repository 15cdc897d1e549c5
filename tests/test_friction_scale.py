"""The friction scale skips its root and quotient where they cannot matter: over random magnitudes, bounds
within a few roundoffs of the root, zeros, denormals, infinities and NaN, it is the plain quotient's bits
wherever that is below 1, and not below 1 wherever that is not."""
import shutil
import struct
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("bits", [32, 64])
def test_friction_scale(bits, tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(ROOT / "physics-engine_gb300" / "csrc"), "-x", "c++",
                    str(ROOT / "tests" / "friction_scale_check.cpp"), "-o", str(exe)], check=True, capture_output=True)
    real = np.float32 if bits == 32 else np.float64
    r = np.random.default_rng(bits)
    n, top = 200000, 44 if bits == 32 else 320
    with np.errstate(all="ignore"):
        q = (10.0 ** r.uniform(-top, top * 0.88, n)).astype(real)
        anyb = (10.0 ** r.uniform(-top, top * 0.88, n)).astype(real)
        root = np.sqrt(q)
        near = root
        for _ in range(3):   # bounds a few roundoffs either side of the root
            near = np.where(r.random(n) < 0.5, np.nextafter(near, real(np.inf)), np.nextafter(near, real(0)))
        wide = (root * (1 + r.normal(0, 1e-5, n))).astype(real)
        odd = np.array([0.0, -0.0, np.inf, np.nan, np.finfo(real).tiny, np.finfo(real).max, 5e-324 if bits == 64 else 1e-45, 1.0, -1.0], real)
        ob, oq = (x.ravel() for x in np.meshgrid(odd, odd))
        b = np.concatenate([anyb, near, wide, np.zeros(n, real), root, -root, ob])
        q = np.concatenate([q] * 6 + [oq])
        want = b / np.sqrt(q)
        (tmp_path / "in").write_bytes(struct.pack("ii", bits, len(b)) + np.stack([b, q], 1).astype(real).tobytes())
        subprocess.run([str(exe), str(tmp_path / "in"), str(tmp_path / "out")], check=True)
        got = np.frombuffer((tmp_path / "out").read_bytes(), real)
        below = want < 1
        assert np.array_equal(below, got < 1)
        whole = np.uint32 if bits == 32 else np.uint64
        assert np.array_equal(want[below].view(whole), got[below].view(whole))
    assert below.any() and not below.all()
