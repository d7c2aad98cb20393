"""Unstaged runs whose solve keeps its values in shared memory.

Blocks of 2 to 6 tiles hold the conjugate gradient's values on the chip
(pearl_fp64.cu, Held): five fields of a cell up to 5 tiles a block, four at 6.
The arithmetic and the order of every sum are the plain kernel's, so each case
equals the oracle in the device's summation order bit for bit.  The cases cover
the smallest and largest of both field counts, one tile below and above the range
(registers, planes), blocks that have a tile less than others, narrow and odd
domains, many iterations (D scaled up), and contexts of different shared-memory
sizes used in turn.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_uniform_tiles import _oracle, _workload

pytestmark = pytest.mark.gpu

GRID = 7
CASES = [
    # nx, ny, D scale (tiles: ceil(nx/32) * ceil(ny/16); a block has tiles/7, rounded up)
    (32, 112, 1.0),  # 7 tiles: one a block
    (32, 113, 1.0),  # 8: two at one block only
    (33, 112, 1.0),  # 14: two at every block
    (70, 163, 100.0),  # 33: five at most, four elsewhere
    (150, 111, 1.0),  # 35: five at every block
    (130, 117, 1.0),  # 40: six at most, five elsewhere
    (96, 223, 100.0),  # 42: six at every block
    (20, 673, 1.0),  # 43: seven at one block, past the range
]


@pytest.fixture
def unstaged(monkeypatch):
    monkeypatch.setenv("PEARL_GPU_TMA", "0")
    monkeypatch.setenv("PEARL_GPU_TILE_WARPS", "8")
    monkeypatch.setenv("PEARL_GPU_GRID", str(GRID))


def _check(port, w, ctx, n):
    g = ctx.geometry()
    assert g["blocks"] == GRID
    phi, carbon, mu, s = ctx.download()
    po, co, muo, so, _ = _oracle(port, w, n, g["warps"], g["blocks"])
    assert np.array_equal(phi, po) and np.array_equal(carbon, co) and np.array_equal(mu, muo)
    assert (s.time, s.dt, s.step, s.rejected) == (so.time, so.dt, so.step, so.rejected)


@pytest.mark.parametrize("nx,ny,dscale", CASES)
def test_bitwise(gpu_lib, port, unstaged, nx, ny, dscale):
    import pearl_gpu

    w = _workload(nx, ny, 24.0, dscale, "layer")
    with pearl_gpu.Context(w.params, nx, ny) as ctx:
        ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        assert ctx.run(3).steps + ctx.run(9).steps == 12
        _check(port, w, ctx, 12)


def test_contexts_in_turn(gpu_lib, port, unstaged):
    """The opt-in for shared memory belongs to the kernel, not to a context: a
    context that holds less does not take it from one that holds more."""
    import pearl_gpu

    cases = [_workload(nx, ny, 24.0, 1.0, None) for nx, ny in ((150, 111), (33, 112), (96, 223))]
    contexts = [pearl_gpu.Context(w.params, w.mu.shape[1], w.mu.shape[0]) for w in cases]
    try:
        for w, ctx in zip(cases, contexts):
            ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        for _ in range(2):
            for ctx in contexts:
                assert ctx.run(3).steps == 3
        for w, ctx in zip(cases, contexts):
            _check(port, w, ctx, 6)
    finally:
        for ctx in contexts:
            ctx.close()


def test_residual_reset(gpu_lib, port, unstaged):
    """A tolerance at the rounding of the residual: the true residual misses it and
    the solve starts again from that."""
    import pearl_gpu

    w = _workload(70, 250, 24.0, 3000.0, "layer")  # 48 tiles: seven a block
    w.params.update(cg_rtol=0.0, cg_atol=5e-18, cg_max=400)
    v = _workload(70, 190, 24.0, 3000.0, "layer")  # 36 tiles: six a block
    v.params.update(cg_rtol=0.0, cg_atol=5e-18, cg_max=400)
    for k in (w, v):
        ny, nx = k.mu.shape
        with pearl_gpu.Context(k.params, nx, ny) as ctx:
            ctx.upload(k.phi, k.carbon, k.mu, k.scalars)
            assert ctx.run(2).steps == 2
            assert ctx.phase_times()["reset"][1] > 0
            _check(port, k, ctx, 2)
