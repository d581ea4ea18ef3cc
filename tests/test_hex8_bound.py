"""The bound that the remelting kernel decides temperatures with (hex8_err32, 2^-19 of the largest node magnitude) holds
for adversarial nodes and coordinates, with the slack of two that its derivation leaves: 15.5 roundings of 2^-24 of that
magnitude are 0.484 of the bound."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("seed", [1, 2])
def test_fp32_interpolation_stays_within_half_its_bound(tmp_path, seed):
    exe = str(tmp_path / "hex8_bound")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", os.path.join(HERE, "hex8_bound.cpp"), "-o", exe],
                   check=True)
    cases, beyond, worst = subprocess.run([exe, "1000000", str(seed)], check=True, capture_output=True,
                                          text=True).stdout.split()
    assert int(cases) >= 1000000 and int(beyond) == 0
    assert 0.02 < float(worst) <= 0.49, worst  # (15.5 * 2^-24 / 2^-19, and the rounding of the largest node itself)
