"""FP64 collide tiles that hold more particles than their staging because the box has
cells enough for all tiles to be resident at once: one collision against the oracle,
both with Philox draws, at the sizes where the rule for the cells per tile turns."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


# 18, 64 and 7 cells per tile (456 tiles in a wave, staging room for 768 particles);
# the last two on the sides of 32 cells: 14,592 = 32 x 456 cells, and more
@pytest.mark.parametrize("L,density", [((20, 20, 20), 100), ((31, 31, 31), 24), ((14, 14, 15), 150),
                                       ((24, 32, 19), 24), ((24, 32, 20), 24)])
def test_fp64_dense_tiles_match_oracle(L, density):
    rng = np.random.default_rng(density + L[2])
    n = density * int(np.prod(L))
    fpos = (rng.random((n, 3)) - 0.5) * np.array(L, float)
    fvel = rng.normal(size=(n, 3))
    o = H.orc.OracleSystem(L, 1.0, 0.1, 1, n)
    o.set_fluid(fpos, fvel)
    o.set_philox(seed=91, counter=3)
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=0.1, h=0.1, seed=91)], precision=capi.FP64,
                      rng=capi.RNG_PHILOX, step_update=1) as ctx:
        ctx.set_fluid(0, fpos, fvel)
        ctx.set_collision_counter(3)
        o.mpc_step(0, 0.1)
        ctx.mpc_step(0, 0.1)
        ctx.raise_on_device_error()
        assert o.error() == 0
        p, v = ctx.get_fluid(0)
    op, ov = o.get_fluid()
    H.close64(p, op)
    H.close64(v, ov)
