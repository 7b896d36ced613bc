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


def test_fp64_cells_of_large_and_outside_coordinates():
    # cell indices come from the coordinate's bits below 2^20 and from a conversion
    # above and below zero: a long box, whose cells the oracle finds by conversion,
    # and strict cells outside the box, which stay an error
    L = (3, 2, 1500)
    rng = np.random.default_rng(8)
    n = 10 * L[0] * L[1] * L[2]
    fpos = (rng.random((n, 3)) - 0.5) * np.array(L)
    fvel = rng.normal(size=(n, 3))
    shift = np.array([0.3, -0.2, 0.1])
    from oracle import oracle as orc
    n_cell = L[0] * L[1] * L[2]
    inj = (shift, rng.gamma(13.5, 1.0, n_cell), rng.random(n_cell), rng.random(n_cell))
    o = orc.OracleSystem(L, 1.0, 0.1, 1, n)
    o.set_fluid(fpos, fvel)
    o.set_inject(*inj)
    o.mpc_step(0, 0.1)
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=0.1, h=0.1)], precision=capi.FP64,
                      rng=capi.RNG_INJECT, step_update=1) as ctx:
        ctx.set_fluid(0, fpos, fvel)
        ctx.mpc_step(0, 0.1, *inj)
        ctx.raise_on_device_error()
        got, _ = ctx.cell_members(0)
        want, _ = o.cell_members()
        np.testing.assert_array_equal(got, want)
        H.close64(ctx.get_fluid(0)[1], o.get_fluid()[1])
