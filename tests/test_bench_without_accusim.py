"""bench.py where accusim cannot be imported: the reference arm says so and ends well, the LJ workloads are built without it."""
import json
import os
import subprocess
import sys

from tests.test_without_accusim import ROOT, SCRIPT

HIDE = SCRIPT[:SCRIPT.index("import devinproj_b200 as b200")]
BODY = """
import bench
import numpy as np
sys.argv = ["bench.py", "--impl", "reference"]
bench.main()
from devinproj_b200 import configs
for name, n in (("argon864", 864), ("lj1m", 1048576)):
    s, forces, dt, cfg = bench.plain_workload(name)
    assert s.n == n == cfg["atoms"] and s.pos.shape == s.vel.shape == (n, 3) and np.all((s.pos >= 0) & (s.pos < s.box))
    T = configs.AR_MASS * np.mean(s.vel ** 2) / configs.k_B
    assert abs(T / (94.4 if n == 864 else 0.72 * 120) - 1) < 5 / np.sqrt(1.5 * n)
    assert np.abs(s.vel.mean(axis=0)).max() < 1e-12 * np.abs(s.vel).max() and s.copy().pos is not s.pos
systems, _, dts, cfg = bench.plain_workload("ensemble")
assert len(systems) == len(dts) == cfg["trajectories"] and sum(x.n for x in systems) == cfg["atoms"]
assert dts[0] == 2 * dts[1] == 4 * dts[2] and np.array_equal(systems[0].vel, systems[2].vel)
"""


def test_bench_without_accusim():
    r = subprocess.run([sys.executable, "-c", HIDE + BODY], cwd=ROOT, capture_output=True, text=True,
                       env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip())
    assert line["impl"] == "reference" and line["unavailable"]
