"""The scan of so many cells that the tiles' totals take a launch of their own (more
than 32,768 tiles of 2,048 cells), against numpy: cell counts and members of a thin
fluid, among them particles in the first and the last cells, after two collisions."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi

pytestmark = pytest.mark.gpu


# 32,768 tiles (two launches), a cell more (three), and a last tile with room
@pytest.mark.parametrize("L", [(512, 512, 256), (512, 257, 511), (421, 409, 397)])
def test_members_of_a_thin_fluid(L):
    rng = np.random.default_rng(L[1])
    n = 200_000
    Lv = np.array(L, float)
    pos = (rng.random((n, 3)) - 0.5) * Lv * 0.999
    pos[:3] = np.array([-0.5, 0.0, 0.5])[:, None] * Lv * 0.9999  # first, middle and last cell
    pos[1] += 0.3
    pos = pos.astype(np.float32).astype(float)
    vel = np.zeros((n, 3))
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=0.0, h=0.0, seed=5)], precision=capi.FP32,
                      rng=capi.RNG_PHILOX, step_update=1, strict_cells=0) as ctx:
        for _ in range(2):  # the counts come back to zero in between
            ctx.set_fluid(0, pos, vel)
            ctx.mpc_bin(0, 0.0, shift=np.zeros(3))
            total, fluid = ctx.cell_counts(0)
            c = np.minimum(np.floor((pos + Lv / 2).astype(np.float32)).astype(int), np.array(L) - 1)
            want = np.bincount(c[:, 0] + L[0] * (c[:, 1] + L[1] * c[:, 2]), minlength=int(np.prod(L)))
            np.testing.assert_array_equal(total, want)
            np.testing.assert_array_equal(fluid, want)
            ctx.mpc_collide()
        ctx.raise_on_device_error()
        got, _ = ctx.get_fluid(0)  # fails when a particle is lost
        np.testing.assert_array_equal(got, pos)
