"""The kernels' division by a constant (csrc/pearl_division.hpp), on the CPU.

a/b is computed as fma(a, zh, a*zl) with two constants per divisor, which the
header proves right for all numerators by trying the few that come near a
rounding boundary.  Here the header is compiled and its quotients are compared
bit for bit with IEEE division: on the divisors of the solver's formulas, on
random ones and on ones with few significant bits, with random numerators of
all signs and sizes, and with numerators next to midpoints that this file finds
by itself with integers.
"""
from __future__ import annotations

import ctypes as C
import math
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "fe-c_eutectoid_phase-field_simulation_b200" / "csrc"

SOURCE = r"""
#include "pearl_division.hpp"
extern "C" int fast_divide(double b, long long n, const double* a, double* q, double* z) {
    double zh, zl;
    const int ok = pearl_gpu::exact_reciprocal(b, zh, zl);
    for (long long i = 0; i < n; ++i) q[i] = std::fma(a[i], zh, a[i] * zl);
    z[0] = zh;
    z[1] = zl;
    return ok;
}
"""

A = (4724862.6373624019, 100000000.0, 172591.65731409981)
FORMULA = [1e-6, 7.1e-6, 2e-9, 2e-9 * 2e-9, 1e-9, 1e-18, 2.5e-9, 2.5e-9 * 2.5e-9, 3.0] + [2.0 * a for a in A]


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    d = tmp_path_factory.mktemp("division")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}",
                    str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    lib = C.CDLL(str(d / "t.so"))
    dp = C.POINTER(C.c_double)
    lib.fast_divide.argtypes = [C.c_double, C.c_longlong, dp, dp, dp]

    def run(b, a):
        a = np.ascontiguousarray(a, dtype=np.float64)
        q, z = np.empty_like(a), np.empty(2)
        ok = lib.fast_divide(b, a.size, a.ctypes.data_as(dp), q.ctypes.data_as(dp), z.ctypes.data_as(dp))
        return bool(ok), q, z

    return run


def _hard(b):
    """Numerators whose quotient by b lies within 32/(2B) ulp of a midpoint."""
    B = int(math.frexp(b)[0] * 2**53)
    t = (B & -B).bit_length() - 1
    Bo = B >> t
    out = []
    if Bo == 1:
        return out
    for s in (53, 54):
        inv = pow(pow(2, s - t, Bo), -1, Bo)
        for n in range(-32, 33):
            if n == 0 or n % (1 << t):
                continue
            a = ((n >> t) * inv) % Bo
            a += -(-(2**52 - a) // Bo) * Bo if a < 2**52 else 0
            while a < 2**53:
                out.append(float(a))
                a += Bo
    return out


def _numerators(rng, n):
    return rng.choice([-1.0, 1.0], n) * rng.uniform(1, 2, n) * 2.0 ** rng.integers(-300, 300, n)


@pytest.mark.parametrize("kind", ["formula", "random", "short"])
def test_quotients_equal_ieee_division(divide, kind):
    rng = np.random.default_rng(5)
    if kind == "formula":
        bs, per = FORMULA, 400000
    elif kind == "random":
        bs, per = rng.uniform(1, 2, 3000) * 2.0 ** rng.integers(-60, 60, 3000), 2000
    else:  # few significant bits: many trailing zeros
        bs, per = [m * 2.0**e for m in range(1, 130) for e in (-20, 0, 30)], 2000
    for b in bs:
        b = float(b)
        a = np.concatenate([_numerators(rng, per), _hard(b), [0.0]])
        ok, q, z = divide(b, a)
        assert ok, b
        assert np.array_equal(q, a / b), b
        assert z[0] == 1.0 / b


def test_odd_divisors_are_refused(divide):
    for b in (0.0, math.inf, math.nan, 5e-324, 1e308 * 1.7):
        with np.errstate(all="ignore"):
            assert not divide(b, [1.0])[0]


def test_zero_and_non_finite_numerators(divide):
    """Zero stays zero and what is not finite stays not finite; the sign of a zero may be lost."""
    for b in FORMULA:
        ok, q, _ = divide(b, [0.0, -0.0, math.inf, -math.inf, math.nan])
        assert ok and q[0] == 0 and q[1] == 0 and not np.isfinite(q[2:]).any()
        assert not np.signbit(q[0])


@pytest.mark.gpu
def test_kernels_of_the_general_division(gpu_lib, port, divide):
    """A molar volume that no constants divide exactly: the kernels compiled with
    the general division, alone and in a batch, against the oracle bit for bit."""
    import os

    import pearl_gpu
    from oracle import pyoracle
    from pearl_gpu import workloads

    vm = next(v for v in (1e-6 * (1.0 + k * 1e-5) for k in range(50000, 70000)) if not divide(v, [1.0])[0])
    w = workloads.scaled(70, 130, seed=4, undercooling=20.0, dt=4e-12, dt_max=8e-12, front=30.0, jitter=0.1)
    w.params["Vm"] = vm
    steps = 5
    with pearl_gpu.Context(w.params, w.nx, w.ny) as ctx:
        ctx.upload(w.phi, w.carbon, w.mu, w.scalars)
        assert ctx.run(steps).steps == steps
        alone, g = ctx.download(), ctx.geometry()
    with pearl_gpu.Batch([(w.params, w.nx, w.ny)]) as b:
        b.configure(g["blocks"], use_tma=False, tile_warps_x=1)
        b.upload(0, w.phi, w.carbon, w.mu, w.scalars)
        assert b.run(steps)[1] == [0]
        batched = b.download(0)
    phi, c, mu = w.phi.copy(), w.carbon.copy(), w.mu.copy()
    s = pyoracle.scalars_from(w.scalars)
    with port.device_order(g["warps"], g["blocks"], g["warps_x_log2"], threads=os.cpu_count()):
        rc, why, k, _ = port.advance_n(w.params, phi, c, mu, s, steps)
    assert rc == 0 and k == steps, why
    for got in (alone, batched):
        assert got[3].time == s.time
        assert all(np.array_equal(a, b) for a, b in zip(got[:3], (phi, c, mu)))
