"""Parts of the solve that the other sizes do not reach, against the oracle (FP64 within the parity bar of
1e-10 and with equal pass counts, mixed within its contract of 1e-5): a full Krylov basis of the largest
restart, an operator cut along k on a slab team, a periodic face that also carries a source, 2D grids of
more rows than one block of the wavefront holds."""
import numpy as np
import pytest

from oracle import run as oracle_run
from radiant_b200 import workloads as W
from radiant_b200._abi import PackedProblem, ResultBuffers

from test_gpu_tiles import check, ctx, grid, settings  # noqa: F401  (ctx: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [60, 61])
def test_largest_restart(ctx, nx):  # noqa: F811
    # 54 mean free paths of nearly pure scattering: GMRES runs through its 48 vectors and restarts
    s = settings(1, 1, 16, 3, restart=48, basis="standard")
    xs = W.synthetic_xs(1, 1, 3, 5)
    xs.sigma_t[:] = 3.0
    xs.sigma_s[:] = 0.0
    for l in range(4):
        xs.sigma_s[0, 0, 0, l] = 2.994 * 0.3 ** l
    tabs = W.slab_tables(nx, np.full(nx, 18.0 / nx), np.ones(nx, dtype=np.int32), 1, 1, 5, s, 3, xs=xs)
    check(ctx, tabs)


@pytest.mark.parametrize("order,precision", [(1, "fp64"), (2, "fp64"), (1, "mixed")])
def test_1d_operator_cut_along_k(ctx, order, precision):  # noqa: F811
    # 140 directions: the D2M operator has 140 columns, more than a CTA's scratch holds of its rows
    s = settings(1, order, 140, 7, basis="standard")
    mats = np.ones(23, dtype=np.int32)
    mats[11:] = 2
    check(ctx, W.slab_tables(23, np.full(23, 4.0 / 23), mats, 2, 2, 5, s, 7, precision=precision))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ns", [(9, 14), (6, 5, 4)])
def test_periodic_face_with_a_source(ctx, ns, precision):  # noqa: F811
    d = len(ns)
    s = settings(d, 1, 4, 2)
    xs = W.synthetic_xs(2, 2, 2, 3)
    mats = np.ones(ns, dtype=np.int32)
    mats[tuple(slice(n // 3, n // 2 + 1) for n in ns)] = 2
    widths = [np.linspace(0.2, 0.3, n) for n in ns]
    beam = ("X-", 0, [1.0, 0.0, 0.0], {a: (0.0, 0.1 * ns[a]) for a in range(1, d)})
    check(ctx, W.grid_tables(d, list(ns), widths, mats, 2, 2, 3, s, 2, beam=beam, bc=(2, 2, 0, 0, 0, 0), precision=precision, xs=xs))


@pytest.mark.parametrize("ns,order,csd,precision", [((4, 257), 2, False, "fp64"), ((5, 290), 2, True, "fp64"), ((6, 300), 1, True, "fp64"),
                                                    ((6, 257), 1, True, "mixed"), ((3, 520), 1, False, "mixed")])
def test_2d_more_rows_than_a_block(ctx, ns, order, csd, precision):  # noqa: F811
    check(ctx, grid(ns, settings(2, order, 4, 2, solver="BFP" if csd else "BTE"), csd=csd, precision=precision, bc=(0, 0, 0, 1, 0, 0)))


@pytest.mark.parametrize("ns", [(1640, 5), (1980, 3, 4)])
def test_dividends_beyond_the_quotients_range(ctx, ns):  # noqa: F811
    # a beam that dies out by 300 orders of magnitude in a pure absorber: the far cells take the division.
    # One moment, one term that outweighs the others in each cell: every cell to 1e-10 of its own value
    d = len(ns)
    s = settings(d, 1, 4, 0, basis="standard")
    xs = W.synthetic_xs(1, 1, 0, 3)
    xs.sigma_t[:] = 6.5
    xs.sigma_s[:] = 0.0
    widths = [np.full(n, 0.2) for n in ns]
    tabs = W.grid_tables(d, list(ns), widths, np.ones(ns, dtype=np.int32), 1, 1, 3, s, 0,
                         beam=("X-", 0, [1.0, 0.0, 0.0], {a: (0.0, 0.2 * ns[a]) for a in range(1, d)}), xs=xs)
    ref = oracle_run.solve(tabs).flux
    pp = PackedProblem(tabs)
    got = ResultBuffers(pp)
    h = ctx.upload(pp)
    ctx.solve(h)
    ctx.download(h, got)
    ctx.release(h)
    assert (np.abs(ref) < 2.0 ** -920).any()
    far = np.abs(ref) > 1e-300
    assert (np.abs(got.flux - ref)[far] <= 1e-10 * np.abs(ref)[far]).all()
