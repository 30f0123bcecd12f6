"""Which 3D problems the octant sweep takes, its offsets into the angular arrays, and the team size of a
launch, on the host."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "radiant.jl_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "libplan.so")
    subprocess.check_call([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                           "--expt-relaxed-constexpr", "--extended-lambda", "-diag-suppress=128", "-I", CSRC,
                           os.path.join(HERE, "native", "plan.cu"), "-o", so])
    lib = ctypes.CDLL(so)
    lib.plan_oct_offset.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("csd", [0, 1])
@pytest.mark.parametrize("mixed", [0, 1])
def test_octant_sweep_takes_large_problems(lib, csd, mixed):
    assert lib.plan_oct3d_ok(64, 64, 64, 80, csd, 148, mixed)
    assert lib.plan_oct3d_ok(416, 192, 192, 288, csd, 148, mixed)  # 4.4e9 angular values, 144 tiles
    assert not lib.plan_oct3d_ok(416, 208, 192, 288, csd, 148, mixed)  # 156 tiles for 148 CTAs


@pytest.mark.parametrize("ns,nd", [((416, 192, 192), 288), ((5, 3, 2), 8), ((100000, 200, 180), 288)])
def test_octant_offsets(lib, ns, nd):
    nx, ny, nz = ns
    for f in range(8):
        for qy, qz, n in [(0, 0, 0), (ny - 1, nz - 1, nd - 1), (1, nz // 2, 3)]:
            iy, iz = qy if f & 2 else ny - 1 - qy, qz if f & 4 else nz - 1 - qz
            ix = 0 if f & 1 else nx - 1
            assert lib.plan_oct_offset(nx, ny, nz, nd, f, qy, qz, n) == nd * (ix + nx * (iy + ny * iz)) + n


FIXED, SERVE, BATCH = 0, 1, 2


@pytest.mark.parametrize("n", [1, 24, 100])
def test_team_size(lib, n):
    # third-order energy closures have no local pass: such slabs keep the caller's size
    for mode in (FIXED, SERVE, BATCH):
        for cluster in (1, 4):
            assert lib.plan_cluster(1, 3, 1, n, cluster, mode) == cluster
    # slabs of the local pass and 2D problems: as many teams as problems, from 4 CTAs up
    want = {1: 16, 24: 8, 100: 4}[n]
    assert lib.plan_cluster(1, 1, 0, n, 4, BATCH) == lib.plan_cluster(2, 1, 0, n, 4, BATCH) == want
    assert lib.plan_cluster(1, 1, 0, n, 2, FIXED) == lib.plan_cluster(2, 1, 0, n, 2, FIXED) == 2
