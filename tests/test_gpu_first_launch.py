"""The device time of a launch (stats) leaves out the loading of its kernel.

A kernel is loaded at its first launch in a process.  That happens before the
event that starts the launch's time, so the first launch of a small domain takes
about as long as the next one on the device: milliseconds less than a load.
"""
from __future__ import annotations

import json
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = """
import json, sys
sys.path.insert(0, "fe-c_eutectoid_phase-field_simulation_b200")
import pearl_gpu
from pearl_gpu import workloads
w = workloads.scaled(64, 48, seed=1, front=12.0)
times = {}
with pearl_gpu.Context(w.params, w.nx, w.ny) as ctx:
    ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
    for name, call in (("run", lambda: ctx.run(1)), ("snapshot", ctx.snapshot), ("mixed", lambda: ctx.run(1))):
        if name == "mixed":
            ctx.set_precision("mixed")
        times[name] = []
        for _ in range(3):
            call()
            times[name].append(ctx.stats()["last_ms"])
with pearl_gpu.Batch([(w.params, w.nx, w.ny)]) as b:
    b.configure(4, use_tma=False)
    b.upload(0, w.phi, w.carbon, w.mu, w.scalars)
    times["batch"] = []
    for _ in range(3):
        b.run(1)
        times["batch"].append(b.stats()["last_ms"])
print(json.dumps(times))
"""


def test_first_launch_time(gpu_lib):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    times = json.loads(r.stdout)
    print(times)
    for name, (first, *later) in times.items():
        assert first < max(later) + 1.0, (name, times)
