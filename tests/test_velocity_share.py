"""The sharing of host-velocity requests between the thread that launched a remelting kernel and its helpers
(amca3d_gb300/csrc/velocity_share.h), with helpers that join late and are descheduled around their loads of the
request word: every entry is evaluated exactly once, before its request counts as answered."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    exe = str(tmp_path_factory.mktemp("share") / "velocity_share")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", os.path.join(HERE, "velocity_share.cpp"), "-o", exe], check=True)
    return lambda scenario, rounds: [int(x) for x in subprocess.run(
        [exe, scenario, str(rounds)], check=True, capture_output=True, text=True, timeout=120).stdout.split()]


@pytest.mark.parametrize("scenario,rounds", [("late", 20), ("late_beside_slow", 5), ("staggered", 8)])
def test_every_entry_is_evaluated_once_before_the_answer(driver, scenario, rounds):
    requests, wrong, unanswered = driver(scenario, rounds)
    assert wrong == 0 and unanswered == 0 and requests == rounds * (400 if scenario == "staggered" else 60)


def test_a_helper_that_does_not_come_back_holds_nobody_beyond_the_launch(driver):
    requests, wrong, unanswered = driver("abandoned", 1)
    assert unanswered == 1 and wrong == 0 and requests >= 1
