"""The FP32 collide on values that no run should hand it: it answers as the kernel of
the strict cells does, and reports what it found and nothing else."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi

pytestmark = pytest.mark.gpu

L = 6
N_CELL = L ** 3


def _fluid(rng, n):
    f32 = lambda a: a.astype(np.float32).astype(np.float64)
    return f32((rng.random((n, 3)) - 0.5) * L), f32(rng.normal(size=(n, 3)))


def _collide(pos, vel, gamma, uphi, utheta, strict=0):
    rep = dict(L=(L,) * 3, n_fluid=len(pos), kT=1.0, shear=0.0, h=0.0, seed=3)
    with capi.Context([rep], precision=capi.FP32, rng=capi.RNG_INJECT, step_update=1, strict_cells=strict) as ctx:
        ctx.set_fluid(0, pos, vel)
        ctx.mpc_step(0, 0.0, np.zeros(3), gamma, uphi, utheta)
        return ctx.error_word()[0], ctx.get_fluid(0)[1]


@pytest.mark.parametrize("bad", [np.nan, -1.0])
def test_a_gamma_variate_without_a_square_root_leaves_the_cell_unscaled(bad):
    rng = np.random.default_rng(5)
    pos, vel = _fluid(rng, 10 * N_CELL)
    gamma, uphi, utheta = rng.gamma(13.5, 1.0, N_CELL), rng.random(N_CELL), rng.random(N_CELL)
    gamma[::3] = bad
    word, v = _collide(pos, vel, gamma, uphi, utheta)
    strict_word, want = _collide(pos, vel, gamma, uphi, utheta, strict=1)
    assert word == strict_word == 0
    # velocities below 8, some ten roundings of 2^-24 each and a factor up to 2
    np.testing.assert_allclose(v, want, rtol=0, atol=2e-5)


# 0: every tile fits its staging; 300: the tile of the first cell does not (360), and
# holds particles that are not a number among the staged ones
@pytest.mark.parametrize("extra", [0, 300])
def test_velocities_that_are_no_numbers_are_reported_as_such_only(extra):
    rng = np.random.default_rng(1)
    pos, vel = _fluid(rng, 10 * N_CELL)
    pos = np.concatenate([pos, (-2.5 + 0.4 * (rng.random((extra, 3)) - 0.5)).astype(np.float32)])
    vel = np.concatenate([vel, rng.normal(size=(extra, 3)).astype(np.float32)])
    bad = np.arange(0, 2000, 50)
    vel[bad] = np.nan
    word, v = _collide(pos, vel, rng.gamma(13.5, 1.0, N_CELL), rng.random(N_CELL), rng.random(N_CELL))
    assert word == 8  # not finite; no term outside the fixed-point range
    assert np.isnan(v[bad]).all()
