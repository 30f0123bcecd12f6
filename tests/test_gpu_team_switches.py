"""RB_LOCAL1D concerns 1D problems: 2D and 3D problems on cluster teams give the same bits with and
without it, and their mixed form runs FP32 passes either way (its result is not the plain form's)."""
import numpy as np
import pytest

from radiant_b200._abi import PackedProblem, ResultBuffers

from test_gpu_local1d import make_ctx
from test_gpu_tiles import grid, settings

pytestmark = pytest.mark.gpu


def solve(ctx, tabs):
    pp = PackedProblem(tabs)
    got = ResultBuffers(pp)
    h = ctx.upload(pp)
    ctx.solve(h)
    ctx.download(h, got)
    ctx.release(h)
    return got.flux.copy()


@pytest.mark.parametrize("ns,csd", [((21, 34), False), ((21, 34), True), ((7, 6, 5), False)])
def test_local1d_switch_leaves_2d_and_3d_alone(ns, csd):
    flux = {}
    for switch in (0, 1):
        ctx = make_ctx(RB_MD_TEAM="cluster", RB_LOCAL1D=switch)
        try:
            for precision in ("fp64", "mixed"):
                flux[switch, precision] = solve(ctx, grid(ns, settings(len(ns), 1, 4, 2, solver="BFP" if csd else "BTE"), csd=csd,
                                                          precision=precision))
        finally:
            ctx.close()
    for precision in ("fp64", "mixed"):
        np.testing.assert_array_equal(flux[0, precision], flux[1, precision])
    assert (flux[0, "mixed"] != flux[0, "fp64"]).any()
