"""wavefront_configure() without arguments gives back the shape that an engine has
which was never configured."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = """
import albedo_b200 as ab
fresh = ab.tuning()
ab.set_tuning(blocks_per_sm=16, trace_blocks_per_sm=2, fetch_batch=64, iterations_per_graph=8, slot_count=1 << 18,
              trace_loop=2, ray_sort=1)
assert ab.tuning() != fresh
ab.wavefront_configure()
assert ab.tuning() == fresh, (ab.tuning(), fresh)
"""


def test_the_defaults_are_a_fresh_engines():
    # In a process of its own: the engine's shape is the process's.
    subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, check=True, timeout=300)
