"""The FP64 products (rb_product.cuh) against a plain loop of FMAs over k, bit for bit: row and column
tiles and their remainders, operators in row blocks and cut along k, both parts, and half of the
directions only (the boundary sums), where a value of the other half must not reach the result even if
it is not finite. The bits hold because mma.sync m8n8k4.f64 adds its four products one after another,
each rounded; the mixed form's results rest on that."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "radiant.jl_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
BIG = 160 << 10  # bytes of a region that holds whole operators


class Sizes(C.Structure):
    _fields_ = [(k, C.c_int) for k in ("ni", "nk", "ncol", "nm", "nmat", "parts", "scaled", "interleave", "sel", "pre", "ncta")] + [
        ("bytes", C.c_longlong), ("alpha", C.c_double)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("product") / "libproduct.so")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                           "-fPIC,-ffp-contract=off", "--extended-lambda", "-I", CSRC, os.path.join(HERE, "native", "product.cu"),
                           "-o", so])
    return C.CDLL(so)


def run(lib, ni, nk, ncol, parts=1, scaled=0, interleave=0, sel=0, pre=0, alpha=1.0, nm=1, ncta=3, region=BIG, stray=None, cut=False):
    z = Sizes(ni, nk, ncol, nm, 3, parts, scaled, interleave, sel, pre, ncta, region, alpha)
    rng = np.random.default_rng(ni + 31 * nk + 101 * ncol)
    A, B = rng.standard_normal((2, nk, ni))
    X = rng.standard_normal((ncol, nk))
    ks, tg = rng.random((3, nk)), rng.random(3)
    mat = rng.integers(0, 3, (ncol + nm - 1) // nm).astype(np.int32)
    selv = rng.standard_normal(ni if sel == 2 else nk)
    P = rng.standard_normal((ncol, ni))
    if stray is not None:
        X[:, selv < 0] = stray
    ptr = [C.c_void_p(a.ctypes.data) for a in (A, B, X, ks, tg, mat, selv, P)]
    got, want = np.full((ncol, ni), 7.0), np.full((ncol, ni), 7.0)
    seg = lib.product_seg(C.byref(z))
    assert (seg > 0) == cut
    lib.product_loop(C.byref(z), *ptr, C.c_void_p(want.ctypes.data), seg)
    assert lib.product_device(C.byref(z), *ptr, C.c_void_p(got.ctypes.data)) == 0
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("ni,nk", [(1, 1), (7, 3), (8, 4), (9, 5), (16, 33), (80, 16), (96, 80), (97, 31), (168, 21)])
@pytest.mark.parametrize("ncol", [1, 8, 9, 700])
def test_one_part(lib, ni, nk, ncol):
    run(lib, ni, nk, ncol)
    run(lib, ni, nk, ncol, scaled=1, pre=1, alpha=-1.0, nm=4)


@pytest.mark.parametrize("ni,nk", [(5, 2), (32, 16), (40, 35), (168, 36)])
@pytest.mark.parametrize("interleave", [0, 1])
def test_two_parts(lib, ni, nk, interleave):
    run(lib, ni, nk, 501, parts=2, scaled=1, interleave=interleave, pre=1, nm=2)


@pytest.mark.parametrize("ni,nk,parts", [(8, 140, 1), (12, 140, 1), (70, 70, 2), (136, 200, 2), (33, 41, 1)])
def test_cut_along_k(lib, ni, nk, parts):
    # the scratch of a team without a region (21504 bytes), and a tighter one
    region = 21504 if nk > 41 else 4800
    run(lib, ni, nk, 77, parts=parts, scaled=1, interleave=1, pre=1, alpha=-1.0, ncta=2, region=region, cut=True)


@pytest.mark.parametrize("ni,nk,region,cut", [(4, 80, BIG, False), (36, 168, BIG, False), (9, 37, BIG, False), (4, 168, 4800, True)])
def test_half_of_the_directions(lib, ni, nk, region, cut):
    run(lib, ni, nk, 301, sel=1, pre=1, alpha=-1.0, region=region, cut=cut)
    run(lib, ni, nk, 301, sel=1, stray=np.nan, region=region, cut=cut)
    run(lib, ni, nk, 301, sel=1, stray=np.inf, region=region, cut=cut)
    run(lib, nk, ni, 301, sel=2)
