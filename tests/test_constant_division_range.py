"""The range of the division by a constant (csrc/pearl_division.hpp), on the CPU.

fma(a, zh, a*zl) equals a/b while a*zl is a normal number, which holds for every
quotient from kExactFrom = 2^-916 up.  The quotients here lie just above that
bound, just below the overflow and anywhere between, and include the numerators
closest to a midpoint.  Below the bound the quotient is within one unit in the
last place, and does miss.
"""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from test_constant_division import CSRC, FORMULA, SOURCE, _hard

SOURCE = SOURCE + 'extern "C" double exact_from() { return pearl_gpu::kExactFrom; }\n'


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("division_range")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{CSRC}",
                    str(d / "t.cpp"), "-o", str(d / "t.so")], check=True)
    lib = C.CDLL(str(d / "t.so"))
    dp = C.POINTER(C.c_double)
    lib.fast_divide.argtypes = [C.c_double, C.c_longlong, dp, dp, dp]
    lib.exact_from.restype = C.c_double
    return lib


def _divide(lib, b, a):
    a = np.ascontiguousarray(a, dtype=np.float64)
    q, z = np.empty_like(a), np.empty(2)
    dp = C.POINTER(C.c_double)
    ok = lib.fast_divide(b, a.size, a.ctypes.data_as(dp), q.ctypes.data_as(dp), z.ctypes.data_as(dp))
    return bool(ok), q, z


def _divisors(rng):
    random = rng.uniform(1, 2, 1500) * 2.0 ** rng.integers(-60, 60, 1500)
    # a reciprocal that a double almost holds: the smallest corrections
    near = [float(np.nextafter(2.0**e * m, s)) for e in (-31, 0, 17) for m in (1.0, 1.25, 1.5) for s in (0.0, np.inf)]
    return [float(b) for b in (*FORMULA, *random, *near)]


@pytest.mark.parametrize("where", ["bound", "top", "between"])
def test_exact_from_the_bound_up(lib, where):
    rng = np.random.default_rng(17)
    low = int(np.log2(lib.exact_from()))
    assert low == -916
    for b in _divisors(rng):
        significands = np.concatenate([rng.uniform(1, 2, 2000), np.asarray(_hard(b)) * 2.0**-52])
        e = {"bound": rng.integers(low, low + 3, significands.size),
             "top": rng.integers(1020, 1024, significands.size),
             "between": rng.integers(low, 1024, significands.size)}[where]
        # the numerator's exponent that gives the quotient's
        shift = e.astype(np.float64) + np.floor(np.log2(b))
        with np.errstate(over="ignore", under="ignore"):
            a = rng.choice([-1.0, 1.0], significands.size) * np.ldexp(significands, shift.astype(int))
            ref = a / b
            use = np.isfinite(ref) & (np.abs(ref) >= lib.exact_from()) & np.isfinite(a) & (np.abs(a) >= 2.0**-1022)
            ok, q, z = _divide(lib, b, a[use])
        if not ok:
            continue  # such a divisor runs the general kernels
        assert np.array_equal(q, ref[use]), b
        if where == "bound":
            assert z[1] == 0 or (np.abs(a[use] * z[1]) >= 2.0**-1022).all(), b


def test_below_the_bound_a_last_place_may_be_missed(lib):
    b = FORMULA[-3]
    rng = np.random.default_rng(18)
    a = np.ldexp(rng.uniform(1, 2, 200000), rng.integers(-1000, -980, 200000))
    ok, q, _ = _divide(lib, b, a)
    ref = a / b
    assert ok and (np.abs(ref) >= 2.0**-1022).mean() > 0.5
    ref, q = ref[np.abs(ref) >= 2.0**-1022], q[np.abs(ref) >= 2.0**-1022]
    missed = q != ref
    assert 0 < missed.mean() < 0.05
    assert (np.abs(q - ref) <= np.spacing(ref)).all()
