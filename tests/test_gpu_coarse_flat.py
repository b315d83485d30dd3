"""Coarse levels at the edges of how the cluster is shared out: levels flat in
x, which it cuts into slabs of y planes where slabs of x planes would not fit,
and levels around the size that its first CTA takes alone.  V-cycles equal the tile
kernels' bit for bit, as in test_gpu_coarse_cluster.py."""
import numpy as np
import pytest

from helpers import assert_bitwise
from test_gpu_coarse_cluster import _vcycle

pytestmark = pytest.mark.gpu

# (grid, levels, precision, level 1 on the cluster): one-plane levels of even and odd extents, a few planes, slabs of
# y planes that divide and that do not, levels on CTA 0 alone below them, a level that fits neither way
GRIDS = [((2, 100, 100), 2, "fp64", True), ((2, 100, 100), 3, "fp32", True), ((3, 120, 110), 3, "fp64", True),
         ((2, 126, 130), 2, "fp32", True), ((2, 128, 128), 3, "fp64", True), ((2, 130, 128), 2, "fp32", True),
         ((4, 200, 64), 3, "fp64", True), ((10, 197, 75), 5, "fp64", True), ((9, 146, 150), 4, "fp32", True),
         ((4, 400, 400), 2, "fp64", False)]
# level 1 on CTA 0 alone in one and in two slots a thread, at the most cells it takes, and one plane above
GRIDS += [(g, 3, p, True) for g in ((24, 24, 24), (32, 16, 16), (32, 16, 32), (34, 16, 32), (34, 16, 16))
          for p in ("fp32", "fp64")]


@pytest.mark.parametrize("grid,levels,prec,coarse", GRIDS)
@pytest.mark.parametrize("sweeps,robust", [((2, 2, 20), True), ((5, 5, 20), False), ((0, 1, 3), True)])
def test_flat_levels_match_tile_kernels(lhi, grid, levels, prec, coarse, sweeps, robust):
    tiles, on_tiles = _vcycle(grid, levels, prec, sweeps, robust, 1)
    joint, on_cluster = _vcycle(grid, levels, prec, sweeps, robust, 0)
    assert not on_tiles and on_cluster == coarse
    assert np.any(joint != 0)
    assert_bitwise(joint, tiles, "z")
