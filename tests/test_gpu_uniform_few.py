"""Mixed-form runs whose uniform tiles belong to a few blocks only.

The FP32 update of the mixed solve walks the whole domain, not a block's own
tiles, so a block needs the value of the uniform tiles although none of its tiles
may be one.  Here a front close below the top wall leaves three to five rows of
uniform tiles (fewer tiles than blocks); a staged run, which leaves them out, is
compared bit for bit with an unstaged one, which does not look for them.  The
chemical potential is uploaded off the composition's by a constant in half of the
cases: the residual of the first solve is then large in the uniform tiles too.
"""
from __future__ import annotations

import numpy as np
import pytest

CASES = [
    # nx, ny, front, rows of tiles that are uniform, offset of mu
    (32, 320, 217.0, 3, 0.0),
    (32, 320, 217.0, 3, 5.0),
    (20, 330, 186.0, 5, 5.0),
    (70, 320, 201.0, 4, 5.0),
]


def _workload(nx, ny, front, offset):
    from pearl_gpu import workloads

    w = workloads.scaled(nx, ny, seed=nx, undercooling=20.0, dt=4e-12, dt_max=8e-12, front=front, jitter=0.1)
    w.mu = np.ascontiguousarray(w.mu + offset)
    return w


def _uniform_rows(w):
    """Tile rows (16 cells) whose cells and neighbours all equal the bulk's reference cell."""
    ny, nx = w.mu.shape
    fields = np.concatenate([w.phi, w.mu[..., None], w.carbon[..., None]], axis=-1)
    same = (fields == fields[ny - 1 - ny // 16, nx // 2]).all(axis=(1, 2))
    rows = -(-ny // 16)
    return sum(bool(same[16 * r - 1:16 * r + 17].all()) for r in range(1, rows - 1))


@pytest.mark.parametrize("nx,ny,front,rows,offset", CASES)
def test_cases_are_what_they_say(nx, ny, front, rows, offset):
    w = _workload(nx, ny, front, offset)
    assert _uniform_rows(w) == rows
    assert rows * -(-nx // 32) < -(-ny // 16) * -(-nx // 32) // 2


def _other(w):
    """Another state of the domain: what it leaves on the chip is not what the case needs."""
    phi, mu = w.phi[:, ::-1].copy(), w.mu + 100.0
    return phi, np.ascontiguousarray(w.carbon[:, ::-1] * 1.01), mu


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "mixed_solve"])
@pytest.mark.parametrize("nx,ny,front,rows,offset", CASES)
def test_context(gpu_lib, monkeypatch, nx, ny, front, rows, offset, precision):
    import pearl_gpu

    w = _workload(nx, ny, front, offset)
    monkeypatch.setenv("PEARL_GPU_TILE_WARPS", "8")
    got = []
    for tma in ("1", "0"):
        monkeypatch.setenv("PEARL_GPU_TMA", tma)
        with pearl_gpu.Context(w.params, nx, ny) as ctx:
            ctx.set_precision(precision)
            ctx.upload(*_other(w), w.scalars)
            try:
                ctx.run(1)
            except pearl_gpu.PearlError:
                pass
            ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
            reports = [ctx.run(k) for k in (1, 4)]
            got.append((ctx.download(), [(r.steps, r.cg_total, r.last.linear_residual) for r in reports]))
    (a, ra), (b, rb) = got
    assert ra == rb and [r[0] for r in ra] == [1, 4]
    assert (a[3].time, a[3].rejected) == (b[3].time, b[3].rejected)
    assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3]))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "mixed_solve"])
@pytest.mark.parametrize("group", [6, 20])
def test_batch(gpu_lib, group, precision):
    import pearl_gpu

    ws = [_workload(nx, ny, front, offset) for nx, ny, front, _, offset in CASES]
    got = []
    for tma in (True, False):
        with pearl_gpu.Batch([(w.params, w.nx, w.ny) for w in ws]) as b:
            b.set_precision(precision)
            b.configure(group, use_tma=tma, tile_warps_x=1)
            for i, w in enumerate(ws):
                b.upload(i, w.phi, w.carbon, w.mu, w.scalars)
            reports, status = b.run(4)
            assert status == [0] * len(ws)
            got.append([(b.download(i), reports[i].cg_total) for i in range(len(ws))])
    for (a, ca), (b, cb) in zip(*got):
        assert ca == cb and a[3].time == b[3].time and a[3].rejected == b[3].rejected
        assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3]))
