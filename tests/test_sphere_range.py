"""The sphere test's early "no root in range" never contradicts the whole test
(tests/cpp/sphere_range.cpp restates both in host arithmetic)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    out = tmp_path_factory.mktemp("sphere") / "sphere_range"
    subprocess.run(["g++", "-std=c++20", "-O2", "-ffp-contract=off", str(HERE / "cpp" / "sphere_range.cpp"), "-o",
                    str(out)], check=True)
    return out


@pytest.mark.parametrize("precision", ["float", "double"])
def test_early_answers_agree_with_the_whole_test(exe, precision):
    lines = subprocess.run([str(exe), precision], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(lines) == 5
    for line in lines:
        tally = {k: int(v) for k, v in (w.split("=") for w in line.split()[1:])}
        assert tally["wrong"] == 0, line
        # The check is not empty: early answers and hits both occur.
        assert tally["early"] > 0.05 * tally["tests"] and tally["hits"] > 0, line
