"""The FP64 collide against the oracle, both with Philox draws, from nearly empty
cells to cells whose particles outgrow the staging of a tile by themselves (768)."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


# particles per cell: tiles of 64 cells up to 10, of 32 from 11 to 21, then fewer, one from 400
@pytest.mark.parametrize("L,density", [(12, 0.3), (12, 2), (12, 10), (9, 11), (8, 21), (8, 23), (6, 60),
                                       (4, 400), (3, 900)])
def test_fp64_collide_matches_oracle_at_every_density(L, density):
    rng = np.random.default_rng(int(10 * density))
    n = int(density * L ** 3)
    fpos = (rng.random((n, 3)) - 0.5) * L
    fvel = rng.normal(size=(n, 3))
    o = H.oracle_for(None, fpos, fvel, L, 1.0, 0.1, 1)
    o.set_philox(seed=91, counter=3)
    with H.context_for(None, fpos, fvel, L, 1.0, 0.1, 1, rng=capi.RNG_PHILOX, seed=91) as ctx:
        ctx.set_collision_counter(3)
        for t in range(3):
            o.mpc_step(t, 0.1)
            ctx.mpc_step(t, 0.1)
        ctx.raise_on_device_error()
        assert o.error() == 0
        p, v = ctx.get_fluid(0)
    op, ov = o.get_fluid()
    # three collisions, each a sum over a cell and a rotation: 1e-12 as every FP64 comparison
    H.close64(p, op)
    H.close64(v, ov)
