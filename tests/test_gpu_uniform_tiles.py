"""Staged runs whose austenite is uniform over whole tiles.

The staged passes leave out the memory traffic of tiles in which every cell
holds the same bits (pearl_fp64.cu, Tiles).  Nothing else may change: each case
is compared bit for bit with the oracle in the device's summation order, on
domains tall enough to hold uniform tiles between the front and the top wall.
The cases cover one tile column and several, a last column that is narrow, wide
or full, both block shapes, a diffusion field that ends inside the domain, a
second bulk value (a window's fill) above the first, more conjugate-gradient
iterations than the dense rim is thick (D scaled up), and a domain without any
uniform tile.
"""
from __future__ import annotations

import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [
    # nx, ny, warps, front, D scale, variant
    (20, 260, 8, 24.0, 1.0, None),
    (33, 300, 8, 24.0, 1.0, None),
    (64, 320, 8, 30.0, 1.0, "layer"),
    (70, 289, 8, 24.0, 1.0, "layer"),
    (150, 400, 8, 60.0, 1.0, "two bulks"),
    (96, 352, 8, 24.0, 400.0, None),
    (45, 350, 8, 24.0, 400.0, "layer"),
    (100, 600, 16, 40.0, 1.0, "layer"),
    (131, 640, 16, 40.0, 1.0, "two bulks"),
    (96, 704, 16, 40.0, 1500.0, None),
    (64, 200, 8, 40.0, 1.0, "all mixed"),
]


def _workload(nx, ny, front, dscale, variant):
    from pearl_gpu import workloads

    w = workloads.scaled(nx, ny, seed=nx + ny, undercooling=20.0, dt=4e-12, dt_max=8e-12, front=front, jitter=0.1,
                         front_jitter=1)
    w.params["D"] = [d * dscale for d in w.params["D"]]
    rows = np.arange(ny)[:, None]
    mu = w.mu
    if variant == "layer":
        mu = mu + 40.0 * np.exp(-((rows - front) / 6.0) ** 2) * np.sin(2 * np.pi * np.arange(nx) / nx)[None, :]
    elif variant == "two bulks":
        mu = np.where(rows < 0.6 * ny, mu, np.nextafter(mu, np.inf))
    elif variant == "all mixed":
        mu = mu + 1e-6 * np.random.default_rng(3).standard_normal((ny, nx))
    chi, c0 = workloads._mixture(w.phi, w.params)
    w.mu = np.ascontiguousarray(mu)
    w.carbon = np.ascontiguousarray(chi * w.mu + c0)
    return w


def _oracle(port, w, n, warps, blocks):
    from oracle import pyoracle

    phi, c, mu = w.phi.copy(), w.carbon.copy(), w.mu.copy()
    s = pyoracle.scalars_from(w.scalars)
    with port.device_order(warps, blocks, 0, threads=os.cpu_count()):
        rc, why, k, infos = port.advance_n(w.params, phi, c, mu, s, n)
    assert rc == 0 and k == n, why
    return phi, c, mu, s, infos


@pytest.mark.parametrize("nx,ny,warps,front,dscale,variant", CASES)
def test_context_bitwise(gpu_lib, port, monkeypatch, nx, ny, warps, front, dscale, variant):
    import pearl_gpu

    monkeypatch.setenv("PEARL_GPU_TMA", "1")
    monkeypatch.setenv("PEARL_GPU_TILE_WARPS", str(warps))
    monkeypatch.setenv("PEARL_GPU_GRID", "7")
    w = _workload(nx, ny, front, dscale, variant)
    n = 6
    with pearl_gpu.Context(w.params, nx, ny) as ctx:
        ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        ctx.set_history(n)
        assert ctx.run(2).steps + ctx.run(n - 2).steps == n
        infos, _ = ctx.history()
        phi, c, mu, s = ctx.download()
        g = ctx.geometry()
    po, co, muo, so, oinfos = _oracle(port, w, n, g["warps"], g["blocks"])
    for f in ("retries", "accepted_dt", "cg_iterations", "linear_residual", "closure", "energy_change"):
        assert [getattr(i, f) for i in infos] == [getattr(i, f) for i in oinfos], f
    if dscale > 1:  # past the rim: 16 cells for 8 warps, 32 for 16
        assert max(i.cg_iterations for i in infos) > 2 * warps
    assert (s.time, s.rejected) == (so.time, so.rejected)
    assert np.array_equal(phi, po) and np.array_equal(c, co) and np.array_equal(mu, muo)


@pytest.mark.parametrize("group", [1, 3])
def test_batch_bitwise(gpu_lib, port, group):
    import pearl_gpu

    ws = [_workload(nx, ny, front, d, v) for nx, ny, warps, front, d, v in CASES if warps == 8]
    n = 4
    with pearl_gpu.Batch([(w.params, w.nx, w.ny) for w in ws]) as b:
        b.configure(group, use_tma=True, tile_warps_x=1)
        for i, w in enumerate(ws):
            b.upload(i, w.phi, w.carbon, w.mu, w.scalars)
        _, st = b.run(n)
        assert st == [0] * len(ws)
        got = [b.download(i) for i in range(len(ws))]
    for w, (phi, c, mu, s) in zip(ws, got):
        po, co, muo, so, _ = _oracle(port, w, n, 8, group)
        assert s.time == so.time
        assert np.array_equal(phi, po) and np.array_equal(c, co) and np.array_equal(mu, muo)


@pytest.mark.parametrize("precision", ["mixed", "mixed_solve", "mixed_propose"])
@pytest.mark.parametrize("nx,ny,warps,front,dscale,variant", CASES)
def test_mixed_forms_equal_dense_runs(gpu_lib, monkeypatch, nx, ny, warps, front, dscale, variant, precision):
    """The mixed forms have no oracle: a staged run, which leaves uniform tiles
    out, against an unstaged one, which does not look for them."""
    import pearl_gpu

    w = _workload(nx, ny, front, dscale, variant)
    monkeypatch.setenv("PEARL_GPU_TILE_WARPS", str(warps))
    monkeypatch.setenv("PEARL_GPU_GRID", "7")
    got = []
    for tma in ("1", "0"):
        monkeypatch.setenv("PEARL_GPU_TMA", tma)
        with pearl_gpu.Context(w.params, nx, ny) as ctx:
            ctx.set_precision(precision)
            ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
            reports = [ctx.run(k) for k in (2, 4)]
            got.append((ctx.download(), [(r.steps, r.cg_total, r.last.linear_residual) for r in reports]))
    (a, ra), (b, rb) = got
    assert ra == rb and sum(r[0] for r in ra) == 6
    assert (a[3].time, a[3].rejected) == (b[3].time, b[3].rejected)
    assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3]))
