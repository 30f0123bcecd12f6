"""The product, sweep and Gram-Schmidt kernels at the edges of their tiles, against the oracle: sizes
around the 8-row and 8-column MMA tiles and 16- and 32-wide wavefronts, odd direction counts, every
2D cell shape with a compiled sweep, row blocks of an operator, restarts. FP64 within 1e-10 relative
L2 (the parity bar: two orders of magnitude above the rounding of the longest sums, N·2^-53 with
N ~ 1e4), mixed within its contract of 1e-5."""
import numpy as np
import pytest

from oracle import run as oracle_run
from radiant_b200 import workloads as W
from radiant_b200._abi import Context, PackedProblem, ResultBuffers
from radiant_b200.sn_flux import SNSettings

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-10, "mixed": 1e-5}


@pytest.fixture(scope="module")
def ctx():
    c = Context(0, 0)
    yield c
    c.close()


def settings(ndims, order, sn, L, solver="BTE", accel="gmres", fc=True, order_e=1, restart=30,
             basis="galerkin-d"):
    axes = ["x", "y", "z"][:ndims] + (["E"] if solver != "BTE" else [])
    orders = {a: (order_e if a == "E" else order) for a in axes}
    return SNSettings(solver_type=solver, quadrature_type="gauss-legendre" if ndims == 1 else "carlson",
                      quadrature_order=sn, legendre_order=L, scheme_type={a: "DD" if o == 1 else "DG" for a, o in orders.items()},
                      scheme_order=orders, acceleration=accel, convergence_criterion=1e-9, maximum_iteration=400,
                      angular_fokker_planck="galerkin", is_full_coupling=fc, gmres_restart=restart,
                      angular_boltzmann=basis)


def grid(ns, sn, ng=2, csd=False, precision="fp64", bc=(0, 0, 0, 0, 0, 0), seed=3):
    mats = np.ones(ns, dtype=np.int32)
    mats[tuple(slice(n // 3, n // 2 + 1) for n in ns)] = 2
    xs = W.synthetic_xs(ng, 2, sn.legendre_order, seed, csd=csd, e_top=2.0, e_cut=2.0 * np.exp(-0.14 * ng))
    widths = [np.linspace(0.2, 0.3, n) for n in ns]  # no two cells of one width
    vol = (0, {a: (0.0, 0.12 * ns[a]) for a in range(len(ns))})
    return W.grid_tables(len(ns), list(ns), widths, mats, ng, 2, seed, sn, sn.legendre_order, volume=vol, bc=bc, csd=csd,
                         precision=precision, xs=xs)


def check(ctx, tabs):
    ref = oracle_run.solve(dict(tabs, precision="fp64"))
    pp = PackedProblem(tabs)
    got = ResultBuffers(pp)
    h = ctx.upload(pp)
    ctx.solve(h)
    ctx.download(h, got)
    ctx.release(h)
    tol = TOL[tabs["precision"]]
    assert np.linalg.norm(got.flux - ref.flux) <= tol * np.linalg.norm(ref.flux)
    if ref.flux_cutoff is not None:
        assert np.linalg.norm(got.flux_cutoff - ref.flux_cutoff) <= tol * np.linalg.norm(ref.flux_cutoff)
    if tabs["precision"] == "fp64":
        assert got.passes == ref.passes


@pytest.mark.parametrize("ns", [(1, 1), (7, 33), (40, 32), (9, 65), (65, 8)])
@pytest.mark.parametrize("csd,precision", [(False, "fp64"), (True, "mixed")])
def test_2d_wavefront_pieces(ctx, ns, csd, precision):
    sn = settings(2, 1, 4, 2, solver="BFP" if csd else "BTE")
    check(ctx, grid(ns, sn, csd=csd, precision=precision, bc=(0, 1, 0, 0, 0, 0)))


@pytest.mark.parametrize("ns", [(5, 3), (13, 33)])
@pytest.mark.parametrize("solver,fc", [("BTE", True), ("BTE", False), ("BFP", True)])
def test_2d_linear_cells(ctx, ns, solver, fc):
    check(ctx, grid(ns, settings(2, 2, 4, 2, solver=solver, fc=fc), csd=solver == "BFP"))


@pytest.mark.parametrize("ns,sn", [((3, 17, 16), 4), ((5, 15, 18), 6), ((100, 4, 5), 2), ((4, 33, 3), 6)])
@pytest.mark.parametrize("csd,precision", [(False, "fp64"), (True, "fp64"), (False, "mixed"), (True, "mixed")])
def test_3d_octant_batches(ctx, ns, sn, csd, precision):
    s = settings(3, 1, sn, 1, solver="BFP" if csd else "BTE", accel="bicgstab")
    check(ctx, grid(ns, s, csd=csd, precision=precision, bc=(0, 0, 0, 0, 1, 0)))


def test_2d_operator_in_row_blocks(ctx):
    # 224 directions, two operator parts: 2 x 224 rows of k do not fit beside all the operator's rows
    check(ctx, grid((6, 5), settings(2, 1, 14, 1, solver="BFP"), ng=1, csd=True))


@pytest.mark.parametrize("nx", [1, 9, 64, 300])
@pytest.mark.parametrize("sn,basis,precision", [(2, "galerkin-d", "fp64"), (10, "galerkin-d", "fp64"), (32, "galerkin-d", "mixed"),
                                                (64, "standard", "fp64"), (64, "standard", "mixed")])
def test_1d_products_and_restarts(ctx, nx, sn, basis, precision):
    s = settings(1, 2, sn, min(sn - 1, 7), solver="BFP", order_e=2, restart=4 if sn < 32 else 30, basis=basis)
    mats = np.ones(nx, dtype=np.int32)
    mats[nx // 2:] = 2
    xs = W.synthetic_xs(3, 2, s.legendre_order, 5, csd=True, e_top=2.0, e_cut=1.3)
    check(ctx, W.slab_tables(nx, np.full(nx, 4.0 / nx), mats, 3, 2, 5, s, s.legendre_order, csd=True, precision=precision, xs=xs))
