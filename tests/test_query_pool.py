"""The workers of host ray queries, on the host against a stand-in for the CUDA
runtime (tests/cpp/query_pool.cpp)."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from albedo_b200.build import CSRC, _cuda_home

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    include = _cuda_home() / "include"
    if shutil.which("g++") is None or not (include / "cuda_runtime_api.h").exists():
        pytest.skip("g++ or the CUDA headers are not available")
    out = tmp_path_factory.mktemp("pool") / "query_pool"
    subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-pthread", f"-I{include}", str(HERE / "cpp" / "query_pool.cpp"),
                    str(CSRC / "query_pool.cpp"), "-o", str(out)], check=True)
    return out


def findings(exe, check):
    """The lines a check prints, as dicts of its numbers; its last line says that nothing is left allocated."""
    lines = subprocess.run([str(exe), check], check=True, capture_output=True, text=True, timeout=120).stdout.splitlines()
    assert lines.pop() == "end left=0"
    return [{k: int(v) for k, v in (w.split("=") for w in line.split()[1:])} for line in lines]


def test_inputs_are_read_after_work_on_the_default_stream(exe):
    found = findings(exe, "order")
    assert [f["count"] for f in found] == [1, 1000, 300_007]
    assert all(f["wrong"] == 0 for f in found), found


def test_a_call_stays_in_its_threads_context(exe):
    found = findings(exe, "context")
    assert [f["own"] for f in found] == [1, 7, 1]
    for f in found:
        assert f["after"] == f["own"] and f["wrong"] == f["elsewhere"] == f["kept_elsewhere"] == 0, found


def test_buffers_stay_while_a_scene_does(exe):
    assert findings(exe, "scenes") == [{"kept": 1, "own_share": 0}]


def test_a_call_runs_with_the_buffers_there_is_memory_for(exe):
    found = findings(exe, "memory")
    assert len(found) == 50
    for f in found:
        assert f["refused"] == (1 if f["limit"] == 0 else 0) and f["wrong"] == f["error"] == 0, f


def test_outputs_over_other_arrays_are_written_after_they_are_read(exe):
    found = findings(exe, "overlap")
    assert len(found) == 30 and all(f["wrong"] == 0 for f in found), found


def test_a_call_that_fails_leaves_nothing_in_flight(exe):
    assert findings(exe, "failure") == [{"bad": bad, "failed": int(bad < 1000), "flight": 0, "wrong": 0}
                                        for bad in (0, 5, -1, 1000)]
