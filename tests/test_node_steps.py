"""The node steps a ray through a mesh is expected to take, by which untuned renders
choose their kernel, on trees done by hand (host, tests/cpp/node_steps.cpp)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "albedo_b200" / "csrc"


@pytest.fixture(scope="module")
def steps(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("steps") / "node_steps"
    host = [str(CSRC / "host" / f"{name}.cpp") for name in ("flatten", "host_scene", "bvh_build", "host_math")]
    subprocess.run(["g++", "-std=c++20", "-O1", "-ffp-contract=off", f"-I{CSRC}", str(HERE / "cpp" / "node_steps.cpp"),
                    *host, "-pthread", "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    return {name: float(value) for name, value in (line.split() for line in lines)}


# Quotients of small whole numbers and powers of two: exact.
@pytest.mark.parametrize("tree,expected", [("empty", 0.0), ("leaf", 1.0), ("tree", 1.625), ("full", 5.0),
                                           ("point", 0.0)])
def test_expected_steps(steps, tree, expected):
    assert steps[tree] == expected
