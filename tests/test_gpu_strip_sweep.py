"""The strip-wise MIC(0) sweeps at the edges of their tiles.

A patch is 16 x 16 lines, a strip 16 x 2; a lane takes two cells of its line per
step and a strip stages chunks of two steps, three or four ahead.  A DOF box spans
whole buckets of 4 cells and at least 16 of them: the blocks below give boxes of 16
lines (one patch), 4 lines more than one patch, 4 fewer than two and three, whole
patches, and 20 to 76 cells along the lines.  The tile wavefront
(WCG_PCG_LAYOUT=tiles) solves the same system with the same recurrences; the pencil
layout's three lower terms are subtracted in another order, so two solves to the
criterion 1e-12 agree to 1e-10 of the largest pressure in FP64 (residual 1e-12
times a condition number below 1e2 at these sizes); in FP32 the coefficients are
rounded to 6e-8 in both and the solves agree to 1e-5."""
import os

import numpy as np
import pytest

from libwetcloth_b200 import _capi, scenes
from libwetcloth_b200.solver import FluidScene

pytestmark = pytest.mark.gpu


def _solve(sc, layout, precision):
    old = os.environ.get("WCG_PCG_LAYOUT")
    os.environ["WCG_PCG_LAYOUT"] = layout
    try:
        g = FluidScene(sc, precision=precision)
    finally:
        if old is None:
            del os.environ["WCG_PCG_LAYOUT"]
        else:
            os.environ["WCG_PCG_LAYOUT"] = old
    g.rebucketize_and_resample()
    g.map_particle_nodes()
    g.step_velocity(1e-3)
    g.project_fine(1e-3)
    p, st = np.nan_to_num(g.field("pressure")), g.stats()
    g.close()
    return p, st


# block extents in cells; the DOF boxes: 16 x 20 x 16, 20 x 20 x 16, 28 x 28 x 32,
# 28 x 56 x 28, 32 x 48 x 32, 44 x 48 x 44, 60 x 20 x 48, 24 x 24 x 76
@pytest.mark.parametrize("cells", [(1, 3, 1), (3, 5, 2), (13, 14, 15), (14, 40, 14), (15, 33, 17),
                                   (30, 31, 29), (46, 6, 31), (7, 9, 62)])
@pytest.mark.parametrize("precision", [_capi.WCG_FP64, _capi.WCG_FP32_REFINE])
def test_strip_edges_match_tiles(cells, precision, wcg):
    n = 64
    sc = scenes.dam_break(n, 8, 9, block_hi=tuple(c / n for c in cells))
    sc.v = np.random.default_rng(3).normal(0.0, 0.2, sc.x.shape)
    sc.params.criterion = 1e-12 if precision == _capi.WCG_FP64 else 1e-8
    a, sa = _solve(sc, "pencil", precision)
    b, sb = _solve(sc, "tiles", precision)
    assert sa["converged"] == 1 and sb["converged"] == 1 and sa["ndof"] == sb["ndof"] > 0
    tol = 1e-10 if precision == _capi.WCG_FP64 else 1e-5
    assert np.abs(a - b).max() <= tol * np.abs(b).max()
    # the same bits again
    c, sc2 = _solve(sc, "pencil", precision)
    assert np.array_equal(a, c) and sa["pcg_iters"] == sc2["pcg_iters"]
