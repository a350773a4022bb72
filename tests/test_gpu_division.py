"""The exact integrator's quotients by a shared reciprocal (recip_rn, div_rn,
div_by) against CUDA's own division, bit for bit, and the recurrences built on
them through both their paths."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SOURCE = os.path.join(ROOT, "tests", "native", "division_check.cu")
LIBRARY = os.path.join(ROOT, "tests", "native", "libdivision_check.so")


def build():
    """The test library, compiled as the exact integrator's unit is."""
    csrc = os.path.join(ROOT, "simcore_b200", "csrc")
    deps = [SOURCE] + [os.path.join(csrc, f) for f in ("sc_step.cuh", "sc_common.cuh", "sc_pair.cuh")]
    if os.path.exists(LIBRARY) and all(os.path.getmtime(LIBRARY) >= os.path.getmtime(p) for p in deps):
        return LIBRARY
    from simcore_b200 import build as product
    subprocess.check_call([product._nvcc()] + product.ARCH +
                          ["-O3", "-std=c++17", "--fmad=false", "-Xcompiler", "-fPIC", "-shared",
                           "-I" + os.path.join(ROOT, "include"), "-I" + csrc, SOURCE, "-o", LIBRARY])
    return LIBRARY


def test_division_check_compiles():
    assert os.path.exists(build())


@pytest.fixture(scope="module")
def lib():
    return ctypes.CDLL(build())


def _ptr(a):
    return a.ctypes.data_as(ctypes.c_void_p)


def _compare(lib, x, b):
    x, b = (np.ascontiguousarray(v, dtype=np.float64) for v in (x, b))
    out = np.full(len(x), -1, dtype=np.int32)
    assert lib.check_given(ctypes.c_int(len(x)), _ptr(x), _ptr(b), _ptr(out)) == 0
    return out


def _mid(v):
    e = (v.view(np.uint64) >> np.uint64(52) & np.uint64(0x7ff)).astype(int) - 1023
    return (e >= -450) & (e < 450)


@pytest.mark.gpu
@pytest.mark.parametrize("exponents", [4, 449])
def test_random_quotients(lib, exponents):
    """2^31 operand pairs, half of them with a quotient near a midpoint between
    two doubles: a narrow range of exponents and the whole range that the fast
    path takes."""
    wrong = ctypes.c_ulonglong(0)
    for seed in (1, 2):
        assert lib.check_random(ctypes.c_ulonglong(seed << 40), ctypes.c_longlong(1 << 30),
                                ctypes.c_int(exponents), ctypes.byref(wrong)) == 0
        assert wrong.value == 0


@pytest.mark.gpu
def test_directed_quotients(lib):
    """Significands of all ones and their neighbours, both ends of the exponents
    that the fast path takes, subnormals, zeros of both signs, infinities and
    NaN: the flag falls exactly where the fast path does not hold, and no
    quotient under it differs."""
    sig = [1.0, 1.0 + 2**-52, 2.0 - 2**-52, 2.0 - 2**-51, 1.5, 4.0 / 3.0, np.nextafter(1.5, 2)]
    exps = [-1022, -451, -450, -449, -1, 0, 1, 448, 449, 450, 451, 1023]
    vals = [s * 2.0**e for s in sig for e in exps]
    vals += [0.0, 5e-324, 2.0**-1040, np.inf, np.nan]
    vals = np.array(vals + [-v for v in vals])
    x, b = (v.ravel() for v in np.meshgrid(vals, vals))
    x, b = x.copy(), b.copy()
    out = _compare(lib, x, b)
    assert not (out & 7).any()
    ones = (b.view(np.uint64) & np.uint64((1 << 52) - 1)) == np.uint64((1 << 52) - 1)
    ok_recip = _mid(b) & ~ones
    assert np.array_equal((out & 8) != 0, ok_recip)
    assert np.array_equal((out & 16) != 0, ok_recip & (_mid(x) | (x == 0)))
    assert ok_recip.any() and (~ok_recip).any()


def _thomas(h, b, d):
    """The reference's tridiagonal_solver (src/linear_algebra.cpp:164-197) with
    symmetric couplings: eliminated diagonal, couplings, solution."""
    m = len(b)
    den, up, v = np.zeros(m), np.zeros(m), np.zeros(m)
    for i in range(m):
        den[i] = b[i] - h[i - 1] * up[i - 1] if i else b[i]
        if i < m - 1:
            up[i] = h[i] / den[i]
        v[i] = (d[i] - h[i - 1] * v[i - 1]) / den[i] if i else d[i] / den[i]
    for i in range(m - 2, -1, -1):
        v[i] = v[i] - up[i] * v[i + 1]
    return den, up[:m - 1], v


def _minors(cz, n, trail):
    """det_t from the tail or det_b from the head (src/filament.cpp:627-660)."""
    out = np.zeros(n + 1)
    x0, x1 = 1.0, 2.0
    at = (lambda i: n - i) if trail else (lambda i: i)
    out[at(0)], out[at(1)] = x0, x1
    for i in range(1, n - 1):
        c = cz[n - 2 - i] if trail else cz[i - 1]
        x0, x1 = x1, 2 * x1 - c * c * x0
        out[at(i + 1)] = x1
    return out


SCALES = {"fast": 1.0, "large": 2.0**460, "small": 2.0**-470}


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 4, 5, 17, 32, 60])
@pytest.mark.parametrize("scale", sorted(SCALES) + ["ones", "late"])
def test_recurrences_take_either_path(lib, n, scale):
    """The elimination, the minors and a right-hand side of one filament, with
    operands that the fast path takes, ones beyond its exponents (the whole
    matrix scaled), a first divisor of all ones, and a last right-hand side
    beyond the exponents: the reference's bits each time."""
    rng = np.random.default_rng(n)
    m = n - 1
    s = SCALES.get(scale, 1.0)
    cz = rng.uniform(0.5, 1.0, 64)
    off = -rng.uniform(0.1, 0.9, 64) * s
    diag = rng.uniform(2.0, 3.0, 64) * s
    d = rng.normal(size=64)
    if scale == "ones":
        diag[0] = 4.0 - 2.0**-51
    if scale == "late":
        d[m - 1] = 2.0**500
    for trail in (0, 1):
        io = np.zeros((9, 64))
        io[0], io[1], io[2], io[7] = cz, off, diag, d
        assert lib.check_solve(_ptr(io), ctypes.c_int(trail), ctypes.c_int(n)) == 0
        h = off[:m] if trail else -cz[:m]
        den, up, x = _thomas(h, diag[:m] if trail else np.full(m, 2.0), d[:m])
        assert np.array_equal(io[3, :m], den)
        assert np.array_equal(io[5, :m - 1], up)
        assert np.array_equal(io[8, :m], x)
        lo = 1 if trail else 0  # det_b[n] .. det_b[1], det_t[0] .. det_t[n - 1]
        assert np.array_equal(io[6, lo:lo + n], _minors(cz, n, trail)[lo:lo + n])
