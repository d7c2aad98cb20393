"""Groups of a batch that are sized per instance, once states are uploaded.

With two blocks an instance or more, and fewer than a block a tile, each instance
gets a group in proportion to the tiles that its passes walk (pearl_batch.cu,
dense_tiles and groups_by_work, restated here).  A group's size is what an
instance's bits depend on, so every case compares each instance bit for bit with
the oracle in the order of the group that it should have: its fields, and the
last step's residual and energy change, in which the order of the sums shows first.
"""
from __future__ import annotations

import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = 296  # 148 SMs x 2 resident blocks
SIZES = [(384, 384), (200, 500), (96, 700)]


def _workloads(fronts, seed=0):
    from pearl_gpu import workloads

    return [workloads.scaled(nx, ny, seed=seed + k, undercooling=14.0 + 3 * k, dt=4e-12, dt_max=8e-12, front=front,
                             jitter=0.1) for k, ((nx, ny), front) in enumerate(zip(SIZES, fronts))]


def _dense(w):
    ny, nx = w.mu.shape
    rows, r = -(-ny // 16), (ny - 1 - ny // 16, nx // 2)
    same = sum(bool((w.phi[16 * k + 8, 0, [0, 2]] == w.phi[r][[0, 2]]).all() and w.mu[16 * k + 8, 0] == w.mu[r]
                    and w.carbon[16 * k + 8, 0] == w.carbon[r]) for k in range(1, rows - 1))
    left_out = max(0, same - 3)
    return -(-nx // 32) * (rows - left_out + 0.05 * left_out)


def _groups(ws):
    """The smallest m for which groups of ceil(dense / m) blocks fit the grid."""
    dense = [_dense(w) for w in ws]
    tiles = [-(-w.nx // 32) * -(-w.ny // 16) for w in ws]

    def sizes(m):
        return [int(max(1.0, min(float(t), math.ceil(d / m)))) for d, t in zip(dense, tiles)]

    lo, hi = 0.0, max(dense)
    for _ in range(40):
        m = 0.5 * (lo + hi)
        lo, hi = (lo, m) if sum(sizes(m)) <= GRID else (m, hi)
    return sizes(hi)


def _upload(batch, ws, only=None):
    for i, w in enumerate(ws):
        if only is None or i in only:
            batch.upload(i, w.phi, w.carbon, w.mu, w.scalars)


def _run(batch, steps):
    reports, status = batch.run(steps)
    assert status == [0] * len(SIZES)
    return reports


def _check(port, batch, reports, i, w, blocks, steps):
    from oracle import pyoracle

    phi, c, mu, s = w.phi.copy(), w.carbon.copy(), w.mu.copy(), pyoracle.scalars_from(w.scalars)
    with port.device_order(8, blocks, 0, threads=os.cpu_count()):
        rc, why, k, infos = port.advance_n(w.params, phi, c, mu, s, steps)
    assert rc == 0 and k == steps, why
    got = batch.download(i)
    assert got[3].time == s.time and got[3].rejected == s.rejected
    for f in ("linear_residual", "closure", "energy_change"):
        assert getattr(reports[i].last, f) == getattr(infos[-1], f), (i, f)
    for a, b in zip(got[:3], (phi, c, mu)):
        assert np.array_equal(a, b), i


@pytest.fixture
def batch(gpu_lib):
    import pearl_gpu

    with pearl_gpu.Batch([(w.params, w.nx, w.ny) for w in _workloads((40.0, 40.0, 40.0))]) as b:
        yield b


LOW, HIGH = (40.0, 200.0, 300.0), (300.0, 60.0, 90.0)


def test_sizes_follow_the_uploaded_states(batch, port):
    assert _groups(_workloads(LOW)) != _groups(_workloads(HIGH))
    for fronts in (LOW, HIGH):
        ws = _workloads(fronts)
        _upload(batch, ws)
        reports = _run(batch, 3)
        sizes = _groups(ws)
        assert batch.stats()["grid"] == sum(sizes)
        for i, w in enumerate(ws):
            _check(port, batch, reports, i, w, sizes[i], 3)


def test_one_new_state_leaves_the_others_their_bits(batch, port):
    ws, new = _workloads(LOW), _workloads(HIGH, seed=5)
    _upload(batch, ws)
    _run(batch, 2)
    sizes = _groups(ws)
    assert _groups([new[0], *ws[1:]]) != sizes
    _upload(batch, new, only=[0])
    reports = _run(batch, 2)
    assert batch.stats()["grid"] == sum(sizes)
    _check(port, batch, reports, 0, new[0], sizes[0], 2)
    for i in (1, 2):
        _check(port, batch, reports, i, ws[i], sizes[i], 4)
    # all of them, in two parts with no run between: a new sweep
    ws = _workloads(HIGH)
    _upload(batch, ws, only=[0, 2])
    _upload(batch, ws, only=[1])
    reports = _run(batch, 2)
    for i, w in enumerate(ws):
        _check(port, batch, reports, i, w, _groups(ws)[i], 2)


def test_autotune_leaves_the_groups_that_run(gpu_lib):
    """On domains large enough for staging to win, and with most of them uniform."""
    import pearl_gpu
    from pearl_gpu import workloads

    ws = [workloads.scaled(nx, ny, seed=k, undercooling=20.0, dt=4e-12, dt_max=8e-12, front=front)
          for k, (nx, ny, front) in enumerate([(640, 1500, 60.0), (512, 1200, 500.0), (400, 1600, 200.0)])]
    tiles = [-(-w.nx // 32) * -(-w.ny // 16) for w in ws]
    sizes = _groups(ws)
    _, planned, _ = pearl_gpu.batch_plan(tiles, GRID, pearl_gpu.BATCH_SIZED_GROUPS)
    assert sum(planned) != sum(sizes)
    with pearl_gpu.Batch([(w.params, w.nx, w.ny) for w in ws]) as b:
        _upload(b, ws)
        # equal groups of up to 16 blocks would leave most of the grid idle
        assert b.autotune(steps=2) == (pearl_gpu.BATCH_SIZED_GROUPS, True, 1)
        timed = b.stats()["grid"]
        _run(b, 2)
        assert timed == b.stats()["grid"] == sum(sizes)


def test_groups_sized_by_tiles_alone_repeat_a_sweep(gpu_lib, port):
    """PEARL_BATCH_SIZED_GROUPS asked for by name: sizes follow the instances' tile
    counts, and a sweep that is downloaded and uploaded again half-way, after the
    fronts have been made to look elsewhere, repeats the uninterrupted one bit for bit."""
    import pearl_gpu

    ws = _workloads(LOW)
    _, sizes, _ = pearl_gpu.batch_plan([-(-nx // 32) * -(-ny // 16) for nx, ny in SIZES], GRID,
                                       pearl_gpu.BATCH_SIZED_GROUPS)
    assert len(sizes) == 3 and list(sizes) != _groups(ws)
    cases = [(w.params, w.nx, w.ny) for w in ws]
    with pearl_gpu.Batch(cases, group_blocks=pearl_gpu.BATCH_SIZED_GROUPS) as b, pearl_gpu.Batch(cases) as c:
        c.configure(pearl_gpu.BATCH_SIZED_GROUPS)
        for batch in (b, c):
            _upload(batch, ws)
            _run(batch, 2)
            half = [batch.download(i) for i in range(3)]
            _upload(batch, _workloads(HIGH))
            _run(batch, 1)
            for i, state in enumerate(half):
                batch.upload(i, *state)
            reports = _run(batch, 2)
            assert batch.stats()["grid"] == sum(sizes)
            for i, w in enumerate(ws):
                _check(port, batch, reports, i, w, int(sizes[i]), 4)
