"""The kernels of the general division on every route that a user reaches.

One parameter set in a hundred has a divisor without exact constants
(exact_reciprocal, csrc/pearl_division.hpp) and runs kernels compiled with the
general division.  Here such a molar volume goes through the staged kernels of both
block shapes (uniform tiles left out), the unstaged ones at one and at several tiles
a block, staged batches, the step without allocation, the mixed forms and the adjoint.  FP64
runs equal the oracle in the device's order bit for bit.
"""
from __future__ import annotations

import ctypes as C
import os

import numpy as np
import pytest

from test_gpu_uniform_tiles import CASES, _oracle, _workload

pytestmark = pytest.mark.gpu

VM = 1.52021e-06  # no neighbour of its reciprocal's correction divides every numerator exactly


def _general(w):
    w.params["Vm"] = VM
    return w


def test_the_volume_has_no_exact_constants():
    from test_constant_division import SOURCE, CSRC
    import subprocess
    import tempfile

    with tempfile.TemporaryDirectory() as d:
        open(f"{d}/t.cpp", "w").write(SOURCE)
        subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}", f"{d}/t.cpp",
                        "-o", f"{d}/t.so"], check=True)
        lib = C.CDLL(f"{d}/t.so")
        dp = C.POINTER(C.c_double)
        lib.fast_divide.argtypes = [C.c_double, C.c_longlong, dp, dp, dp]
        z = (C.c_double * 2)()
        assert not lib.fast_divide(VM, 0, z, z, z)


@pytest.mark.parametrize("tma", ["1", "0"])
@pytest.mark.parametrize("nx,ny,warps,front,dscale,variant", CASES)
def test_context_bitwise(gpu_lib, port, monkeypatch, nx, ny, warps, front, dscale, variant, tma):
    import pearl_gpu

    monkeypatch.setenv("PEARL_GPU_TMA", tma)
    monkeypatch.setenv("PEARL_GPU_TILE_WARPS", str(warps))
    monkeypatch.setenv("PEARL_GPU_GRID", "7")
    w = _general(_workload(nx, ny, front, dscale, variant))
    with pearl_gpu.Context(w.params, nx, ny) as ctx:
        ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        assert ctx.run(2).steps + ctx.run(2).steps == 4
        phi, c, mu, s = ctx.download()
        g = ctx.geometry()
    po, co, muo, so, _ = _oracle(port, w, 4, g["warps"], g["blocks"])
    assert (s.time, s.rejected) == (so.time, so.rejected)
    assert np.array_equal(phi, po) and np.array_equal(c, co) and np.array_equal(mu, muo)


def test_batch_bitwise(gpu_lib, port):
    """One such instance decides for the whole batch: the others keep their bits."""
    import pearl_gpu

    ws = [_workload(nx, ny, front, d, v) for nx, ny, warps, front, d, v in CASES if warps == 8]
    for w in ws[::2]:
        _general(w)
    with pearl_gpu.Batch([(w.params, w.nx, w.ny) for w in ws]) as b:
        b.configure(3, use_tma=True, tile_warps_x=1)
        for i, w in enumerate(ws):
            b.upload(i, w.phi, w.carbon, w.mu, w.scalars)
        assert b.run(4)[1] == [0] * len(ws)
        got = [b.download(i) for i in range(len(ws))]
    for w, (phi, c, mu, s) in zip(ws, got):
        po, co, muo, so, _ = _oracle(port, w, 4, 8, 3)
        assert s.time == so.time
        assert np.array_equal(phi, po) and np.array_equal(c, co) and np.array_equal(mu, muo)


@pytest.mark.parametrize("precision", ["mixed", "mixed_solve", "mixed_propose"])
@pytest.mark.parametrize("nx,ny,warps,front,dscale,variant", CASES[2::3])
def test_mixed_forms_equal_dense_runs(gpu_lib, monkeypatch, nx, ny, warps, front, dscale, variant, precision):
    import pearl_gpu

    w = _general(_workload(nx, ny, front, dscale, variant))
    monkeypatch.setenv("PEARL_GPU_TILE_WARPS", str(warps))
    got = []
    for tma in ("1", "0"):
        monkeypatch.setenv("PEARL_GPU_TMA", tma)
        with pearl_gpu.Context(w.params, nx, ny) as ctx:
            ctx.set_precision(precision)
            ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
            assert ctx.run(4).steps == 4
            got.append(ctx.download())
    a, b = got
    assert a[3].time == b[3].time and all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3]))


def test_step_without_allocation(gpu_lib, port):
    import pearl_gpu
    import torch

    w = _general(_workload(70, 130, 30.0, 1.0, "layer"))
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (np.moveaxis(w.phi, -1, 0), w.carbon, w.mu)]
    p, s, info = (pearl_gpu.PearlParams.from_dict(w.params), pearl_gpu.PearlScalars.from_dict(w.scalars),
                  pearl_gpu.PearlStepInfo())
    tiles = -(-70 // 32) * -(-130 // 16)
    for _ in range(2):
        rc = gpu_lib.pearl_gpu_advance_noalloc(C.byref(p), 70, 130, *(C.c_void_p(t.data_ptr()) for t in dev), C.byref(s),
                                               1e300, C.byref(info), None)
        assert rc == 0
    po, co, muo, so, _ = _oracle(port, w, 2, 8, tiles)
    assert s.time == so.time
    assert np.array_equal(np.moveaxis(dev[0].cpu().numpy(), 0, -1), po)
    assert np.array_equal(dev[1].cpu().numpy(), co) and np.array_equal(dev[2].cpu().numpy(), muo)


def test_adjoint(gpu_lib, port):
    from oracle import pyoracle
    import pearl_gpu
    from pearl_gpu import workloads

    steps = 40
    w = _general(workloads.adjoint_case(64, 96, pairs=1, steps=steps, front=24.0))
    target = np.ascontiguousarray(w.phi[..., 0] * 0.9)
    with pearl_gpu.Context(w.params, w.nx, w.ny) as ctx:
        ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        rep = ctx.adjoint_gradient(steps, 15, target)
    rc, orep = port.adjoint_gradient(w.params, w.phi.copy(), w.carbon.copy(), w.mu.copy(),
                                     pyoracle.scalars_from(w.scalars), steps, 15, target)
    assert rc == 0
    assert rep.objective == pytest.approx(orep.objective, rel=1e-8)
    for k in range(3):
        assert rep.grad[k] == pytest.approx(orep.grad[k], rel=1e-4)
