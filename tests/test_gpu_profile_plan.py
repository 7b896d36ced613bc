"""Velocity profiles on both sides of the sizes where the runs per thread lengthen
(311,296, 622,592, 1,245,184 and 2,490,368 slots) and where the sums go into copies of
the bins (300 particles per bin), against numpy."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi
from tests.test_gpu_readout import _profile

pytestmark = pytest.mark.gpu

# edges, solvent particles, width
CASES = [((8, 8, 8), 1, 1.0), ((8, 8, 8), 2699, 1.0), ((8, 8, 8), 2700, 1.0),   # 18 bins: copies from 2,700
         ((11, 9, 8), 5200, 0.02),                                              # many bins, one copy
         ((16, 16, 16), 129, 0.5), ((32, 32, 32), 311_295, 1.0), ((32, 32, 32), 311_296, 1.0),
         ((32, 32, 32), 311_296, 0.02), ((40, 40, 40), 622_593, 0.01), ((50, 50, 50), 1_245_184, 0.05),
         ((60, 60, 60), 2_490_369, 1.0), ((60, 60, 60), 2_490_369, 0.003)]


@pytest.mark.parametrize("precision", [capi.FP32, capi.FP64], ids=["fp32", "fp64"])
@pytest.mark.parametrize("L,n,width", CASES, ids=[f"{c[0][0]}-{c[1]}-{c[2]}" for c in CASES])
def test_profile_of_every_plan(precision, L, n, width):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) - 0.5) * np.asarray(L, float)
    vel = rng.normal(size=(n, 3))
    if precision == capi.FP32:
        pos, vel = (a.astype(np.float32).astype(np.float64) for a in (pos, vel))
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=0.1, h=0.1, seed=3)], precision=precision,
                      rng=capi.RNG_PHILOX, step_update=1, strict_cells=0) as ctx:
        ctx.set_fluid(0, pos, vel)
        ctx.set_delrx(0, 0.7)
        for _ in range(2):  # the bins start from zero each time
            got = ctx.velocity_profile(0, width)
            for g, w in zip(got, _profile(pos, vel, L, 0.1, 0.7, width)):
                np.testing.assert_array_equal(g[:, 2], w[:, 2])
                # sums of up to n terms of size ~5: n eps times that
                np.testing.assert_allclose(g[:, :2], w[:, :2], rtol=0, atol=n * 5 * 2.3e-16 * 4)
