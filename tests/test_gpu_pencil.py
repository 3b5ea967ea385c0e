"""The pressure solve in the pencil layout against the tile wavefront.

Both layouts run the same MIC(0)-PCG arithmetic (the order of the three
lower-neighbour terms and the products sent across patch edges can round
differently), so pressures agree to 1e-10 relative to their maximum in FP64
and iteration counts agree to one.  The scenes cover each axis as the stream
axis and boxes spanning several patches along both cut axes (patch edges and
the tagged edge words between patches)."""
import os

import numpy as np
import pytest

from libwetcloth_b200 import _capi, scenes
from libwetcloth_b200.solver import FluidScene

pytestmark = pytest.mark.gpu
DT = 1e-3


def _scene(kind):
    if kind == "dam16_y":
        return scenes.dam_break(16, 8, 0)
    if kind == "slab64_x":
        return scenes.dam_break(64, 2, 3, block_hi=(0.9, 0.3, 0.6))
    if kind == "slab48_z":
        return scenes.dam_break(48, 2, 4, block_hi=(0.5, 0.3, 0.95))
    if kind == "curl48":
        return scenes.half_box(48, 2, 5, amplitude=0.5, sigma_cells=2.0)
    raise ValueError(kind)


def _solve(sc, layout, precision, groups=None):
    """The pressure and the solver's figures; groups: the groups per cluster of
    the sweeps (None: chosen by the box)."""
    env = {"WCG_PCG_LAYOUT": layout}
    if groups is not None:
        env["WCG_SWEEP_CL"] = str(groups)
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        g = FluidScene(sc, precision=precision)
    finally:
        for k, v in old.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v
    g.rebucketize_and_resample()
    g.map_particle_nodes()
    g.step_velocity(DT)
    g.project_fine(DT)
    p = g.field("pressure")
    st = g.stats()
    # extents of the DOF box (fields are bucket-major, 4 x 4 x 4 nodes a bucket)
    dims, _, _ = g.grid_info()
    dof = np.flatnonzero(g.ifield("dof_index") >= 0)
    b, n = dof // 64, dof % 64
    xyz = [4 * (b % dims[0]) + n % 4, 4 * (b // dims[0] % dims[1]) + n // 4 % 4,
           4 * (b // (dims[0] * dims[1])) + n // 16]
    st["box"] = [int(k.max() - k.min()) + 1 for k in xyz]
    g.close()
    return p, st


@pytest.mark.parametrize("kind", ["dam16_y", "slab64_x", "slab48_z", "curl48"])
def test_pencil_matches_tiles_fp64(kind, wcg):
    sc = _scene(kind)
    p_pl, st_pl = _solve(sc, "pencil", _capi.WCG_FP64)
    p_t, st_t = _solve(sc, "tiles", _capi.WCG_FP64)
    assert st_pl["converged"] == 1 and st_t["converged"] == 1
    assert abs(st_pl["pcg_iters"] - st_t["pcg_iters"]) <= 1, (st_pl, st_t)
    m = ~np.isnan(p_t)
    assert np.array_equal(m, ~np.isnan(p_pl))
    scale = np.abs(p_t[m]).max()
    assert np.abs(p_pl[m] - p_t[m]).max() <= 1e-10 * scale
    assert st_pl["residual"] <= sc.params.criterion * st_pl["rhs_norm"]


@pytest.mark.parametrize("kind", ["slab64_x", "curl48"])
def test_pencil_matches_tiles_fp32_refine(kind, wcg):
    sc = _scene(kind)
    p_pl, st_pl = _solve(sc, "pencil", _capi.WCG_FP32_REFINE)
    p_t, st_t = _solve(sc, "tiles", _capi.WCG_FP32_REFINE)
    assert st_pl["converged"] == 1 and st_t["converged"] == 1
    m = ~np.isnan(p_t)
    scale = np.abs(p_t[m]).max()
    assert np.abs(p_pl[m] - p_t[m]).max() <= 1e-5 * scale
    assert st_pl["residual"] <= sc.params.criterion * st_pl["rhs_norm"]


def test_pencil_deterministic(wcg):
    sc = _scene("curl48")
    a, sa = _solve(sc, "pencil", _capi.WCG_FP32_REFINE)
    b, sb = _solve(sc, "pencil", _capi.WCG_FP32_REFINE)
    assert sa["pcg_iters"] == sb["pcg_iters"]
    m = ~np.isnan(a)
    assert np.array_equal(a[m], b[m])


@pytest.mark.parametrize("precision", [_capi.WCG_FP32_REFINE, _capi.WCG_FP64])
def test_pencil_deterministic_256_patches(precision, wcg):
    """The 256^3 half box (256 patches, more than the SMs hold at one CTA
    each): three solves of the same system give the same pressures and
    iteration counts bit for bit."""
    sc = scenes.half_box(256, 2, seed=1)
    res = []
    for _ in range(3):
        g = FluidScene(sc, precision=precision)
        g.set_correction_count(0)
        g.rebucketize_and_resample()
        g.map_particle_nodes()
        g.step_velocity(DT)
        g.project_fine(DT)
        st = g.stats()
        res.append((np.nan_to_num(g.field("pressure")), st["pcg_iters"], st["refinements"]))
        g.close()
    for p, it, rf in res[1:]:
        assert it == res[0][1] and rf == res[0][2]
        assert np.array_equal(p, res[0][0])


def _groups(box, precision):
    """(groups in a column of patches, groups in all) of a DOF box: 16 x 16 lines
    a patch across its longest axis, one group a patch in FP32 and two in FP64."""
    s = box.index(max(box))
    a, c = [k for k in range(3) if k != s]
    col = -(-box[c] // 16) * (1 if precision == _capi.WCG_FP32_REFINE else 2)
    return col, col * -(-box[a] // 16)


# blocks of liquid (cells) whose boxes have 1, 2, 3, 5 and more groups in a column
# (multiples of 4 and not), and 74 groups at most or more in all
@pytest.mark.parametrize("cells,precision,column,many", [
    ((20, 40, 2), _capi.WCG_FP32_REFINE, 1, False),
    ((20, 40, 10), _capi.WCG_FP32_REFINE, 2, False),
    ((24, 60, 24), _capi.WCG_FP32_REFINE, 3, False),
    ((30, 70, 58), _capi.WCG_FP32_REFINE, 5, False),
    ((100, 130, 118), _capi.WCG_FP32_REFINE, 9, False),
    ((130, 140, 118), _capi.WCG_FP32_REFINE, 9, True),
    ((20, 40, 2), _capi.WCG_FP64, 2, False),
    ((20, 60, 24), _capi.WCG_FP64, 6, False),
    ((30, 70, 58), _capi.WCG_FP64, 10, False),
    ((78, 100, 74), _capi.WCG_FP64, 12, False),
    ((90, 100, 74), _capi.WCG_FP64, 12, True),
])
def test_sweeps_in_clusters_and_without_bit_identical(cells, precision, column, many, wcg):
    """Clusters only change how the c-face values of a group travel (shared memory
    of the next CTA in place of a global round trip): the sweeps in clusters of 4
    groups, those without and the form that the box's size chooses give the same
    pressures and iteration counts bit for bit, also where the groups of a column
    are not a multiple of 4."""
    n = 160
    sc = scenes.dam_break(n, 2, 9, block_hi=tuple(c / n for c in cells))
    sc.v = np.random.default_rng(3).normal(0.0, 0.2, sc.x.shape)
    a, sa = _solve(sc, "pencil", precision, 1)
    col, groups = _groups(sa["box"], precision)
    assert col == column and (groups > 74) == many, (sa["box"], col, groups)
    assert sa["converged"] == 1
    m = ~np.isnan(a)
    for g in (4, None):
        b, sb = _solve(sc, "pencil", precision, g)
        assert sa["pcg_iters"] == sb["pcg_iters"] and sa["refinements"] == sb["refinements"]
        assert np.array_equal(m, ~np.isnan(b)) and np.array_equal(a[m], b[m])
