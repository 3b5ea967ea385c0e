"""The multigrid's smoothing at odd and ragged extents.

A thread relaxes the cell of its colour in a pair along x and walks further
pairs when a level has more of them than a launch has threads.  The boxes below
have levels of odd and even extents, of fewer pairs than one block and of more
than one launch holds.  The preconditioner decides how many iterations a solve
takes, so a cell left out shows there; the solution is that of the MIC(0)
solver: both stop at a residual of 1e-10, and with a condition number of about
1e4 (a box of 130 cells) the pressures agree to 1e-6 of the largest (1e-5 in
FP32, whose coefficients are rounded to 6e-8)."""
import numpy as np
import pytest

from libwetcloth_b200 import _capi, scenes
from libwetcloth_b200.solver import FluidScene

pytestmark = pytest.mark.gpu


def _solve(cells, precision, mg):
    n = max(cells)
    sc = scenes.dam_break(n, 2, 4, block_hi=tuple(c / n for c in cells))
    sc.v = 0.3 * np.sin(7.0 * sc.x[:, [1, 2, 0]])
    sc.params.criterion = 1e-10 if precision == _capi.WCG_FP64 else 1e-8
    solver = _capi.WCG_SOLVER_MG if mg else _capi.WCG_SOLVER_MIC0
    g = FluidScene(sc, precision=precision, solver=solver)
    g.rebucketize_and_resample()
    g.map_particle_nodes()
    g.step_velocity(1e-3)
    g.project_fine(1e-3)
    p, st = np.nan_to_num(g.field("pressure")), g.stats()
    g.close()
    assert st["converged"] == 1
    return p, st["pcg_iters"]


@pytest.mark.parametrize("cells", [(3, 2, 5), (17, 9, 14), (33, 31, 40), (131, 67, 129)])
@pytest.mark.parametrize("precision", [_capi.WCG_FP64, _capi.WCG_FP32_REFINE])
def test_levels_match_mic0(cells, precision, wcg):
    a, ia = _solve(cells, precision, True)
    b, ib = _solve(cells, precision, False)
    tol = 1e-6 if precision == _capi.WCG_FP64 else 1e-5
    assert np.abs(a - b).max() <= tol * np.abs(b).max()
    assert ia <= max(ib, 4)
