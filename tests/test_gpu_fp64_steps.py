"""The FP64 quotients and reciprocal square roots of csrc/fp64_steps.cuh, over the exponents and at zero,
subnormal, infinite and NaN operands.  Each ends in one FMA (half a unit in the last place) of terms whose
own errors are below one unit, so 2 units of the exact value (in extended precision) bound them; operands
that they pass to CUDA's operators give the operators' results."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "nnpp-mg-implant-corrosion-3d_gb300", "csrc")
DIV_NEWTON, DIV_CORRECTED, RSQRT_NEWTON, RSQRT_STEP = range(4)


@pytest.fixture(scope="module")
def steps(nn, tmp_path_factory):
    if nn.device_count() < 1:
        pytest.skip("no CUDA device")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("fp64_steps") / "libsteps.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler", "-fPIC",
                    "-shared", "-I", CSRC, os.path.join(HERE, "fp64_steps_check.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def run(op, a, b=None):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ascontiguousarray(np.ones_like(a) if b is None else b, dtype=np.float64)
        out, cuda = np.empty_like(a), np.empty_like(a)
        ptr = [x.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for x in (a, b, out, cuda)]
        assert lib.fp64_steps(op, a.size, *ptr) == 0
        return out, cuda

    return run


def _values(rng, n, e0, e1):
    """Random significands and signs with exponents spread over [e0, e1], and the powers of two's neighbours."""
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(e0, e1 + 1, n)) * rng.choice([-1.0, 1.0], n)
    p = np.ldexp(1.0, np.arange(e0, e1 + 1))
    return np.concatenate([x, p, np.nextafter(p, 0), np.nextafter(p, np.inf)])


def _units(out, exact):
    return (np.abs(out.astype(np.longdouble) - exact) / np.spacing(np.abs(exact.astype(np.float64)))).max()


def _same(out, cuda):
    return np.array_equal(out, cuda, equal_nan=True) and np.array_equal(np.signbit(out), np.signbit(cuda)) \
        if not np.isnan(cuda).any() else np.array_equal(out, cuda, equal_nan=True)


SPECIAL = np.array([0.0, -0.0, 5e-324, -5e-324, 2.2e-308, 1e-300, -1.0, 3.0, 1.7976931348623157e308, np.inf, -np.inf,
                    np.nan])


def test_div_newton(steps):
    rng = np.random.default_rng(1)
    b = _values(rng, 200000, -1022, 1021)
    # quotients in the normal range
    e = np.clip(rng.integers(-900, 901, b.size), -900 - np.frexp(b)[1], 900 - np.frexp(b)[1])
    a = np.ldexp(rng.uniform(1.0, 2.0, b.size), np.clip(e + np.frexp(b)[1], -950, 1000))
    exact = a.astype(np.longdouble) / b.astype(np.longdouble)
    keep = (np.abs(exact) > 1e-290) & (np.abs(exact) < 1e290)
    out, _ = steps(DIV_NEWTON, a, b)
    assert keep.sum() > 100000
    assert _units(out[keep], exact[keep]) <= 2
    a, b = (x.ravel() for x in np.meshgrid(SPECIAL, SPECIAL))
    out, cuda = steps(DIV_NEWTON, a, b)
    exact_ops = (np.abs(a) < 1e-288) | ~np.isfinite(a) | (np.abs(b) < 2.3e-308) | ~np.isfinite(b)
    assert _same(out[exact_ops], cuda[exact_ops])
    assert np.allclose(out, cuda, rtol=4.5e-16, atol=0.0, equal_nan=True)


def test_div_corrected(steps):
    rng = np.random.default_rng(2)
    d = _values(rng, 200000, -490, 490)
    a = _values(rng, 400000, -520, 520)[:d.size]
    exact = a.astype(np.longdouble) / d.astype(np.longdouble)
    keep = (np.abs(exact) > 1e-290) & (np.abs(exact) < 1e290)
    out, _ = steps(DIV_CORRECTED, a, d)
    assert keep.sum() > 100000
    assert _units(out[keep], exact[keep]) <= 2
    a, d = (x.ravel() for x in np.meshgrid(SPECIAL, np.array([1e-140, -3e-4, 0.1, 7.0, 1e140])))
    out, cuda = steps(DIV_CORRECTED, a, d)
    finite = np.isfinite(cuda)
    assert np.array_equal(out[~finite], cuda[~finite], equal_nan=True)
    assert (np.abs(out[finite] - cuda[finite]) <= 2 * np.spacing(np.abs(cuda[finite]))).all()
    assert np.array_equal(np.signbit(out[finite]), np.signbit(cuda[finite]))


@pytest.mark.parametrize("op,e0,e1", [(RSQRT_NEWTON, -1022, 1023), (RSQRT_STEP, -110, 110)])
def test_rsqrt(steps, op, e0, e1):
    x = np.abs(_values(np.random.default_rng(3), 400000, e0, e1))
    out, _ = steps(op, x)
    assert _units(out, 1 / np.sqrt(x.astype(np.longdouble))) <= 2
    x = SPECIAL[~(SPECIAL < 0)] if op == RSQRT_NEWTON else SPECIAL
    x = x[~((x == 0) & np.signbit(x))]
    out, cuda = steps(op, x)
    assert np.allclose(out, cuda, rtol=4.5e-16, atol=0.0, equal_nan=True)
