"""The coarse levels solved by one thread-block cluster against the tile
kernels (one launch per colour, restriction and prolongation by the tile
kernels), which the limit ``coarse_cells`` selects for every level.

Both update every cell with the same arithmetic in the same order on the
same values, so V-cycles agree bit for bit on every cell with a row.
The grids put the slabs' edges everywhere they can fall: fewer planes than
CTAs, planes that do not divide, odd extents (uncovered fine cells, ragged
rows), levels that run on the cluster, on one CTA, or on both.
"""
import numpy as np
import pytest

from liquidhairinteration_b200 import abi, scenes
from liquidhairinteration_b200.model import LiquidModel

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

# (grid, levels): the finest coarse level's extents are the halves
GRIDS = [((16, 16, 16), 2), ((32, 32, 32), 3), ((64, 64, 64), 4), ((66, 30, 34), 4), ((93, 70, 61), 4),
         ((23, 62, 90), 3), ((128, 24, 40), 5), ((12, 12, 12), 4)]


def _vcycle(grid, levels, prec, sweeps, robust, coarse_cells):
    flags = dict(scenes.ROBUST_SOLVER if robust else scenes.REFERENCE_SOLVER)
    solver = abi.make_solver_params(**{**flags, "num_level": levels, "num_pre_smooth": sweeps[0],
                                       "num_post_smooth": sweeps[1], "num_final_smooth": sweeps[2],
                                       "coarse_cells": coarse_cells})
    h = 1.0 / grid[0]
    m = LiquidModel.from_params(abi.make_grid_desc(grid, (0, 0, 0), tuple(n * h for n in grid)), solver,
                                abi.make_liquid_params(), prec)
    rng = np.random.default_rng(5)
    x, y, z = np.meshgrid(*[np.arange(n) for n in grid], indexing="ij")
    phi = (y - 0.6 * grid[1] + 2.0 * np.sin(0.3 * x) + rng.uniform(-1.5, 1.5, size=grid)) * h
    phi[rng.uniform(size=grid) < 0.01] = 0.0
    m.set_field("liquidPhi", phi)
    for a, name in enumerate("xyz"):
        shape = list(grid)
        shape[a] += 1
        w = rng.uniform(0.2, 1.0, size=shape) * (rng.uniform(size=shape) < 0.9)
        m.set_field("liquidW" + name, w)
        m.set_field("v" + name, rng.standard_normal(shape))
    s = m.GetSolver()
    s.Init()
    s.BuildRHS()
    s.BuildLHS(1000.0, 1.0 / 480.0)
    m.set_field("r", m.field("rhs") * (m.field("liquidPhi") <= 0))
    s.ApplyPreconditioner()
    s.ApplyPreconditioner()  # a second cycle, from the first's z
    out, coarse = m.field("z"), s.ActiveTiles(1)[2]
    wet = m.field("liquidPhi") <= 0
    m.close()
    return out[wet], coarse


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("grid,levels", GRIDS)
@pytest.mark.parametrize("sweeps,robust", [((2, 2, 20), True), ((5, 5, 20), False), ((0, 1, 3), True)])
def test_cluster_vcycle_matches_tile_kernels(lhi, grid, levels, prec, sweeps, robust):
    tiles, on_tiles = _vcycle(grid, levels, prec, sweeps, robust, 1)
    joint, on_cluster = _vcycle(grid, levels, prec, sweeps, robust, 0)
    assert not on_tiles
    n1 = [g // 2 for g in grid]
    slab = -(-n1[0] // 16) * n1[1] * (-(-n1[2] // 2))  # cells of one colour in a CTA's slab of level 1
    assert on_cluster == (slab <= (2048 if prec == "fp32" else 1024))
    assert np.any(joint != 0)
    assert_bitwise(joint, tiles, "z")
