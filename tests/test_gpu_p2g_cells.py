"""P2G with chosen numbers of particles in a cell and in a row of cells, at the
edges of the sizes its warps stage at once (24 particles), against the oracle.
Tolerance (FP32): a face sums at most 27 cells of 97 particles, and an order of
summation changes a sum of n positive terms by at most n units of 2^-24 --
2600 * 2^-24 = 1.6e-4 in the worst case, sqrt(n) of that kind of error in the
mean: 2e-5 of the largest weight; the velocities divide two such sums."""
import numpy as np
import pytest

from liquidhairinteration_b200 import scenes

from helpers import assert_close, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("counts", [(1,), (23, 1), (24,), (24, 1), (25, 23, 48), (49, 0, 97, 1, 24, 24, 7, 2)])
def test_p2g_particle_counts(oracle_mod, lhi, prec, counts):
    g, o = pair(oracle_mod, scenes.dam(16), prec, with_particles=False)
    dt = np.float64 if prec == "fp64" else np.float32
    rng = np.random.default_rng(31)
    cells = []
    for x, y, z in ((2, 3, 0), (2, 3, 6), (7, 8, 7), (15, 15, 8)):  # over a tile's edges and at the grid's
        cells += [((x, y, (z + k) % 16), c) for k, c in enumerate(counts)]
    pos = np.concatenate([(np.array(c) + rng.uniform(0.02, 0.98, (n, 3))) / 16 for c, n in cells]).astype(dt)
    vel = rng.uniform(-1, 1, pos.shape).astype(dt)
    aff = rng.uniform(-5, 5, (len(pos), 9)).astype(dt)
    g.GetParticleSystem().SetParticles(pos, vel, aff)
    o.set_particles(pos, vel, aff)
    g.clear()
    g.Particle2Grid()
    o.clear()
    o.particle_to_grid()
    rtol = 1e-12 if prec == "fp64" else 2e-5
    for f in ("wx", "wy", "wz"):
        assert_close(g.field(f), o.field(f), rtol, rtol * np.abs(o.field(f)).max(), f)
    for f in ("vx", "vy", "vz"):
        a, b, w = g.field(f), o.field(f), o.field("w" + f[1])
        far = w > 1e-3 * w.max()  # elsewhere the quotient is of two small sums
        assert_close(a[far], b[far], rtol * 10, rtol * 10 * np.abs(b[far]).max(), f)
