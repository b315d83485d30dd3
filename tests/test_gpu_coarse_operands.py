"""The coarse cluster's quotients and sums outside the ordinary range, against
the tile kernels (``coarse_cells`` = 1): V-cycles on residuals near and below
the least normal number, near the largest, with infinities and NaN, and on
diagonals too large for the stored reciprocal.

Both form every value by the same roundings, and neither reads a neighbour
that is not in the row, so they agree bit for bit, and on where the result
is not a number: infinities of one pool do not reach the other.
"""
import numpy as np
import pytest

from liquidhairinteration_b200 import abi, scenes
from liquidhairinteration_b200.model import LiquidModel

pytestmark = pytest.mark.gpu

GRID, LEVELS = (40, 48, 64), 4


def _vcycle(prec, sweeps, robust, coarse_cells, density, scale, odd, w=None):
    flags = dict(scenes.ROBUST_SOLVER if robust else scenes.REFERENCE_SOLVER)
    solver = abi.make_solver_params(**{**flags, "num_level": LEVELS, "num_pre_smooth": sweeps[0],
                                       "num_post_smooth": sweeps[1], "num_final_smooth": sweeps[2],
                                       "coarse_cells": coarse_cells, **({} if w is None else {"smoothing_factor": w})})
    h = 1.0 / GRID[0]
    m = LiquidModel.from_params(abi.make_grid_desc(GRID, (0, 0, 0), tuple(n * h for n in GRID)), solver,
                                abi.make_liquid_params(), prec)
    rng = np.random.default_rng(5)
    x, y, z = np.meshgrid(*[np.arange(n) for n in GRID], indexing="ij")
    # two pools with a gap of two coarsest cells between them, one at each end of the rows: next to each other in
    # memory and no neighbours
    phi = np.maximum(y - 0.6 * GRID[1] + 2.0 * np.sin(0.3 * x), 8.0 - np.abs(z - 31.5)) * h
    m.set_field("liquidPhi", phi)
    for a, name in enumerate("xyz"):
        shape = list(GRID)
        shape[a] += 1
        m.set_field("liquidW" + name, rng.uniform(0.2, 1.0, size=shape) * (rng.uniform(size=shape) < 0.9))
    s = m.GetSolver()
    s.Init()
    s.BuildRHS()
    s.BuildLHS(density, 1.0 / 480.0)
    wet = phi <= 0
    with np.errstate(over="ignore", under="ignore"):
        r = (np.ldexp(rng.standard_normal(GRID), scale + rng.integers(-8, 9, size=GRID)) * wet).astype(m.dtype)
    if odd:
        first = np.argwhere(wet & (z < 24))
        for k, v in enumerate((np.inf, -np.inf, np.nan)[:odd]):
            r[tuple(first[(2 * k + 1) * len(first) // 7])] = v
    m.set_field("r", r)
    s.ApplyPreconditioner()
    s.ApplyPreconditioner()  # a second cycle, from the first's z
    out, coarse, d = m.field("z").reshape(GRID), s.ActiveTiles(1)[2], np.abs(m.field("Adiag")).reshape(GRID)
    m.close()
    return out[wet], out[wet & (z > 40)], coarse, d[wet].max()


def _compare(prec, sweeps, robust, density, scale, odd=0, w=None):
    tiles, far_tiles, on_tiles, _ = _vcycle(prec, sweeps, robust, 1, density, scale, odd, w)
    joint, far_joint, on_cluster, d = _vcycle(prec, sweeps, robust, 0, density, scale, odd, w)
    assert on_cluster and not on_tiles
    if odd:
        assert np.isfinite(far_tiles).all() and np.any(far_tiles != 0)
        # (without a sweep on the finest level one infinity can end in coarse cells that have no row)
        assert not np.isfinite(tiles).all() or (odd == 1 and sweeps[:2] == (0, 0))
    nan = np.isnan(tiles)
    assert np.array_equal(np.isnan(joint), nan), (int(np.isnan(joint).sum()), int(nan.sum()))
    bits = np.uint32 if joint.dtype == np.float32 else np.uint64
    differ = joint[~nan].view(bits) != tiles[~nan].view(bits)
    assert not differ.any(), (int(differ.sum()), joint[~nan][differ][:4], tiles[~nan][differ][:4])
    if odd:
        assert np.array_equal(far_joint.view(bits), far_tiles.view(bits))
    return joint, d


SWEEPS = [((2, 2, 20), True), ((5, 5, 20), False), ((0, 1, 3), True), ((0, 0, 1), True)]


@pytest.mark.parametrize("prec,scale", [("fp32", k) for k in (-85, -100, -118, -128, -140, 112, 118)] +
                         [("fp64", k) for k in (-890, -950, -1010, -1050, 1005, 1012)])
@pytest.mark.parametrize("sweeps,robust", SWEEPS)
def test_small_and_large_residuals(lhi, prec, scale, sweeps, robust):
    joint, _ = _compare(prec, sweeps, robust, 1000.0, scale)
    assert np.any(joint != 0)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("odd", [1, 2, 3])
@pytest.mark.parametrize("sweeps,robust", SWEEPS)
def test_infinities_and_nan(lhi, prec, odd, sweeps, robust):
    _compare(prec, sweeps, robust, 1000.0, 0, odd)


# diagonals on both sides of the largest that divide by their reciprocal (2^26, 2^100), and near the largest number
@pytest.mark.parametrize("prec,density", [("fp32", 4e-7), ("fp32", 1e-34), ("fp64", 4e-29), ("fp64", 1e-300)])
@pytest.mark.parametrize("sweeps,robust", SWEEPS)
def test_large_diagonals(lhi, prec, density, sweeps, robust):
    joint, d = _compare(prec, sweeps, robust, density, 0)
    assert np.any(joint != 0)
    assert np.isfinite(d) and d > (2.0 ** 26 if prec == "fp32" else 2.0 ** 100)


# a factor whose products round, in both smoothers
@pytest.mark.parametrize("prec,scale", [("fp32", 0), ("fp64", 0), ("fp32", -128), ("fp64", -1050)])
@pytest.mark.parametrize("sweeps,robust", SWEEPS)
def test_smoothing_factor(lhi, prec, scale, sweeps, robust):
    _compare(prec, sweeps, robust, 1000.0, scale, w=0.7)
