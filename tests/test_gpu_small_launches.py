"""The collision's bookkeeping at the edges of its launch shapes: cell counts around
what one CTA scans (8,192) and around tiles of 2,048, solvent counts around the
binning tiles (512 to 4,096 slots), and the delrx advance inside the collision."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi

pytestmark = pytest.mark.gpu

# edges, solvent particles
BOXES = [((1, 1, 1), 1), ((8, 8, 8), 511), ((8, 8, 8), 513), ((16, 16, 8), 1025), ((16, 16, 16), 4097),
         ((32, 16, 16), 20000), ((33, 16, 16), 20000), ((32, 32, 10), 1024 * 40), ((31, 17, 23), 70001),
         ((64, 64, 32), 312000), ((64, 64, 33), 313000)]


@pytest.mark.parametrize("precision", [capi.FP64, capi.FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("L,n", BOXES, ids=[f"{a}x{b}x{c}-{n}" for (a, b, c), n in BOXES])
def test_every_particle_is_sorted_and_momentum_is_kept(L, n, precision):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) - 0.5) * np.array(L) * 0.999
    vel = rng.normal(size=(n, 3))
    if precision == capi.FP32:
        pos, vel = pos.astype(np.float32).astype(float), vel.astype(np.float32).astype(float)
    shear, h = 0.7, 0.1
    rep = dict(L=L, n_fluid=n, n_mono=0, mol0_size=0, kT=1.0, shear=0.0, h=h, md_dt=0.01, seed=5)
    kw = dict(precision=precision, rng=capi.RNG_PHILOX, step_update=10, delrx_mode=capi.DELRX_PHYSICAL)
    with capi.Context([rep], **kw) as ctx:
        ctx.set_fluid(0, pos, vel)
        ctx.cycles(3)
        ctx.raise_on_device_error()
        _, v = ctx.get_fluid(0)  # fails when a particle is lost
    # velocities of order one in sums of n: FP64 round-off, FP32 a unit of 2^-23 each per collision
    tol = n * (1e-13 if precision == capi.FP64 else 3 * 2.0 ** -21)
    np.testing.assert_allclose(v.sum(axis=0), vel.sum(axis=0), rtol=0, atol=tol)
    # the same box sheared: delrx as the reference advances it, ten times a cycle
    with capi.Context([dict(rep, shear=shear)], **kw) as ctx:
        ctx.set_fluid(0, pos, vel)
        ctx.cycles(7)
        ctx.raise_on_device_error()
        got = ctx.delrx(0)
    want = 0.0
    for _ in range(70):
        want += shear * L[1] * (h * (1.0 / 10))
        want -= L[0] * np.copysign(np.floor(abs(want / L[0]) + 0.5), want)
    assert got == want
