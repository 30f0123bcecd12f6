"""The sweeps' quotient (rb_quot.cuh) against the plain division, on the host and on the device, over
the whole exponent range with zeros, infinities and NaN.

Inside its range the method is within half a unit in the last place and a trace of q/s (2^-50 of a
unit in FP64, 2^-22 in FP32), the division within half a unit: they differ by at most one unit, and
only where q/s lies within the trace of the middle of two numbers, which in FP64 fewer than one random
pair in 2^49 does. Outside the range the quotient is the division itself. So: one unit at most, and
no difference on random FP64 pairs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "radiant.jl_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quotients") / "libquotients.so")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-shared", "-Xcompiler",
                           "-fPIC,-ffp-contract=off", "-I", CSRC, os.path.join(HERE, "native", "quotients.cu"), "-o", so])
    return ctypes.CDLL(so)


def quotients(lib, q, s, device):
    got, want = np.empty_like(q), np.empty_like(q)
    f = lib.quotients_f64 if q.dtype == np.float64 else lib.quotients_f32
    ptr = [a.ctypes.data_as(ctypes.c_void_p) for a in (q, s, got, want)]
    assert f(*ptr, len(q), int(device)) == 0
    return got, want


def draws(dtype, n=1 << 20):
    """Pairs over all exponents, pairs in the sweeps' range, and every pair of the special values."""
    rng = np.random.default_rng(7)
    fi = np.finfo(dtype)

    def vals(lo, hi):
        m = (1.0 + rng.random(n)).astype(dtype) * np.where(rng.random(n) < 0.5, -1, 1).astype(dtype)
        return np.ldexp(m, rng.integers(lo, hi, n)).astype(dtype)

    b = (900, 100) if dtype == np.float64 else (90, 30)  # the range's ends
    low = fi.minexp - fi.nmant
    edge = [np.ldexp(dtype(m), e).astype(dtype) for e in (-b[0], b[0] - 1, b[0], -b[1], b[1] - 1, b[1], fi.minexp, low, fi.maxexp - 1, 0)
            for m in (1.0, 1.0 + 2 * float(fi.eps), 2.0 - float(fi.eps))]
    sp = np.array(edge + [0.0, np.inf, np.nan, 3e-308 if dtype == np.float64 else 3e-38, 0.37], dtype=dtype)
    sp = np.concatenate([sp, -sp])
    qs, ss = (a.ravel() for a in np.meshgrid(sp, sp))
    q = np.concatenate([vals(low, fi.maxexp), vals(-b[0], b[0]), vals(-20, 20), qs])
    s = np.concatenate([vals(low, fi.maxexp), vals(-b[1], b[1]), vals(-20, 20), ss])
    return np.ascontiguousarray(q), np.ascontiguousarray(s), 3 * n


def check(lib, dtype, device):
    with np.errstate(all="ignore"):
        q, s, nrand = draws(dtype)
        got, want = quotients(lib, q, s, device)
        same = (got.view(f"i{got.itemsize}") == want.view(f"i{got.itemsize}")) | (np.isnan(got) & np.isnan(want))
        if dtype == np.float64:
            assert same[:nrand].all()
        near = np.isfinite(got) & np.isfinite(want) & (np.abs(got - want) <= np.spacing(np.abs(want)))
        assert (same | near).all(), [(a, b, c, d) for a, b, c, d in zip(q, s, got, want)][: 5]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_quotients_host(lib, dtype):
    check(lib, dtype, False)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_quotients_device(lib, dtype):
    check(lib, dtype, True)
