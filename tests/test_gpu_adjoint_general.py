"""The reverse step's general solve (pearl_adjoint.cuh, adj_solve).

A domain of more than two cells a thread solves with its vectors in the planes;
below that they stay in registers.  With a grid limited to a few blocks small
domains take the general solve too.  The gradient is held to the CPU reference
gradient, and to the one from the solve in registers: the same arithmetic in
another order of the sums.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 40


def _case(nx, ny, pairs):
    from pearl_gpu import workloads

    w = workloads.adjoint_case(nx, ny, pairs=pairs, steps=STEPS, front=24.0)
    return w, np.ascontiguousarray(w.phi[..., 0] * 0.9)


def _gradient(w, target, every):
    import pearl_gpu

    with pearl_gpu.Context(w.params, w.nx, w.ny) as ctx:
        ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        rep = ctx.adjoint_gradient(STEPS, every, target)
        return rep, ctx.geometry()["blocks"]


@pytest.mark.parametrize("nx,ny,pairs,grid", [
    (64, 96, 1, 11),  # 6144 cells on 11 blocks of 256: some threads a third cell
    (64, 96, 1, 1),
    (97, 65, 2, 3),   # odd, 8.2 cells a thread
    (64, 96, 1, 12),  # two cells a thread: the last domain in registers
])
def test_gradient(gpu_lib, port, monkeypatch, nx, ny, pairs, grid):
    from oracle import pyoracle

    w, target = _case(nx, ny, pairs)
    registers, blocks = _gradient(w, target, 15)
    assert nx * ny <= 2 * 256 * blocks
    monkeypatch.setenv("PEARL_GPU_GRID", str(grid))
    rep, blocks = _gradient(w, target, 15)
    assert blocks == grid and (nx * ny > 2 * 256 * grid) == (grid != 12)
    rc, orep = port.adjoint_gradient(w.params, w.phi.copy(), w.carbon.copy(), w.mu.copy(),
                                     pyoracle.scalars_from(w.scalars), STEPS, 15, target)
    assert rc == 0
    assert rep.steps == STEPS and rep.objective == pytest.approx(orep.objective, rel=1e-8)
    for k in range(3):
        assert rep.grad[k] == pytest.approx(orep.grad[k], rel=1e-4)
        # two solves to the same relative tolerance 1e-11 a step, 40 steps
        assert rep.grad[k] == pytest.approx(registers.grad[k], rel=1e-8)
    again, _ = _gradient(w, target, 15)
    assert list(again.grad) == list(rep.grad)
