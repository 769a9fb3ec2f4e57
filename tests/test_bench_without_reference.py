"""bench.py where the reference renderer is absent: the reference arm prints one line
that says so and succeeds, on rank 0 alone, and the errors against it are marked
unavailable (host).
"""

import importlib.util
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

from oracle import reference as ref

BENCH = Path(__file__).resolve().parent.parent / "bench.py"

pytestmark = pytest.mark.skipif(ref.available(), reason="the reference library is here")


@pytest.mark.parametrize("rank", [0, 1])
def test_reference_arm_says_it_is_unavailable(rank):
    env = {"RANK": str(rank), "LOCAL_RANK": str(rank), "WORLD_SIZE": "2"} if rank else {}
    done = subprocess.run([sys.executable, str(BENCH), "--impl", "reference", "--gpus", str(rank + 1), "--steps", "20",
                           "--warmup", "5"], capture_output=True, text=True, timeout=300, env={**os.environ, **env})
    assert done.returncode == 0, done.stderr
    lines = [json.loads(line) for line in done.stdout.splitlines() if line.strip()]
    assert [set(line) for line in lines] == ([{"impl", "unavailable"}] if rank == 0 else [])
    assert all(line["impl"] == "reference" and line["unavailable"] for line in lines)


def test_errors_against_the_reference_are_unavailable(tmp_path):
    spec = importlib.util.spec_from_file_location("bench_under_test", BENCH)
    bench = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = bench
    spec.loader.exec_module(bench)
    assert set(bench.precision_errors(tmp_path / "absent.scene", bench.LARGE, {})) == {"unavailable"}
