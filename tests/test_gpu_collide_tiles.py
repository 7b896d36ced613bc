"""FP32 collide tiles at the edges of their size rule and staging capacity:
one collision from identical inputs and draws against the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc
from starpolymersmd_gb300 import capi, system
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


# n_c = 1, 3: tiles of at most 32 cells far below the staging capacity; 10:
# tiles near it; 20, 45: fewer cells per tile. `extra` particles in one cell
# beside a star's core send that tile past the capacity of 360, with monomers
# among the particles that are read from global memory again.
@pytest.mark.parametrize("L,n_c,extra", [(5, 1, 0), (9, 3, 0), (11, 10, 0), (11, 10, 55), (11, 10, 700),
                                         (7, 20, 0), (7, 20, 200), (6, 45, 0), (6, 45, 400), (21, 10, 330)])
def test_fp32_collide_tile_edges(L, n_c, extra):
    rng = np.random.default_rng(100 * L + n_c)
    f32 = lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)
    fpos, fvel = system.uniform_fluid((L,) * 3, n_c, 1.0, rng)
    if extra:
        fpos = np.concatenate([fpos, 0.5 + 0.4 * (rng.random((extra, 3)) - 0.5)])
        fvel = np.concatenate([fvel, rng.normal(size=(extra, 3))])
    fpos, fvel = f32(fpos), f32(fvel)
    star = None
    for _ in range(200):
        star = system.make_star(3, 2, 0.5, 5.0, 1.0, rng, bond=0.97, anchor_bond=1.2, outward_bias=0.0)
        if np.abs(star.pos).max() < L / 2 - 0.9:
            break
    star.pos, star.vel = f32(star.pos), f32(star.vel)
    n_cell, shear, h = L ** 3, 0.03, 0.1
    shift = f32(rng.random(3) - 0.5)
    gamma, uphi, uth = (f32(a) for a in (rng.gamma(1.5 * max(1, n_c - 1), 1.0, n_cell),
                                         rng.random(n_cell), rng.random(n_cell)))
    # the oracle's forces do not act here (no MD substeps); wrapped binning
    o = orc.OracleSystem((L,) * 3, 1.0, shear, 1, len(fpos), star.n, mol_start=[0, star.n],
                         delrx_dt_scale=1.0, mono_wrap=1)
    o.set_fluid(fpos, fvel)
    o.set_monomers(star.pos, star.vel, np.zeros_like(star.pos), np.full(star.n, 5.0), star.amphi,
                   star.anchor)
    o.set_inject(shift, gamma, uphi, uth)
    o.mpc_step(0, h)
    assert o.error() == 0
    rep = dict(L=(L,) * 3, n_fluid=len(fpos), n_mono=star.n, mol0_size=star.n, kT=1.0, shear=shear,
               h=h, seed=3)
    with capi.Context([rep], precision=capi.FP32, rng=capi.RNG_INJECT, step_update=1, strict_cells=0,
                      mono_bin=capi.MONOBIN_WRAPPED, delrx_mode=capi.DELRX_PHYSICAL) as ctx:
        ctx.set_fluid(0, fpos, fvel)
        ctx.set_monomers(0, star.pos, star.vel, np.zeros_like(star.pos), np.full(star.n, 5.0),
                         star.amphi, star.anchor)
        ctx.mpc_step(0, h, shift, gamma, uphi, uth)
        ctx.raise_on_device_error()
        H.fp32_cycle_check(ctx, o, 0, L)
