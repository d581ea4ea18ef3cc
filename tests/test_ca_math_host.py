"""The envelope arithmetic of the CUDA kernels (amca3d_gb300/csrc/ca_math.h),
compiled for the host with the same no-contraction rule, against the
reference Octahedron known answers (tests/golden/kat_octahedron.npz)."""
import os
import shutil
import struct
import subprocess
import tempfile

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_ca_math_matches_reference_octahedron():
    k = np.load(os.path.join(HERE, "golden", "kat_octahedron.npz"))
    inp = k["inputs"]
    n = len(inp)
    gc = inp[:, 6:9] - inp[:, 3:6]
    rows = np.concatenate([k["l2g"], gc, inp[:, 9:11], k["trunc"][:, None],
                           k["captured"][:, None].astype(np.float64), k["info"]], axis=1)
    assert rows.shape == (n, 20)
    with tempfile.TemporaryDirectory() as wd:
        exe = os.path.join(wd, "kat")
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "ca_math_kat.cpp"),
                        "-o", exe], check=True)
        data = os.path.join(wd, "kat.bin")
        with open(data, "wb") as f:
            f.write(struct.pack("<i", n))
            f.write(rows.astype("<f8").tobytes())
        out = subprocess.run([exe, data], check=True, capture_output=True, text=True).stdout.split()
    total, caps, bad = map(int, out)
    assert total == n and caps == int(k["captured"].sum()) and bad == 0


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_capture_equals_the_general_path_and_helpers_the_fp64_operations(tmp_path):
    """Ordinary captures, zeros and ties, near ties, lengths over the exponent range and points on the surface:
    capture_f64 returns capture_f64_general's bits; each helper its FP64 operation's."""
    exe = str(tmp_path / "paths")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "capture_paths.cpp"), "-o", exe],
                   check=True)
    out = subprocess.run([exe, "200000", "7"], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [line.split() for line in out if line]
    assert len(rows) == 13 and all(int(n) == 200000 and int(wrong) == 0 for _, n, wrong in rows), rows


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_capture_with_any_truncation_equals_the_general_path(tmp_path):
    """Truncations with a sign, NaN, infinities and products that underflow (an envelope evaluation takes any):
    capture_f64 returns capture_f64_general's bits."""
    exe = str(tmp_path / "truncation")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "capture_truncation.cpp"), "-o", exe],
                   check=True)
    rows = [line.split() for line in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()]
    assert len(rows) == 13 and all(int(wrong) == 0 for _, _, wrong in rows), rows
