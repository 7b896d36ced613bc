"""The FP32 collide's results do not depend on how a box is cut into tiles: the same box
alone and beside empty boxes, which change the cells per tile (8, 15 and 29 or 30), with
a crowded cell that fits its tile's staging in the first cut and outgrows it in the
others, and a star's monomers among its particles."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi, system, workloads as W

pytestmark = pytest.mark.gpu

L = 11


def _run(beside, extra, cycles=3):
    rng = np.random.default_rng(12)
    f32 = lambda a: np.asarray(a, dtype=np.float32).astype(np.float64)
    fpos, fvel = system.uniform_fluid((L,) * 3, 10, 1.0, rng)
    fpos = f32(np.concatenate([fpos, 0.5 + 0.4 * (rng.random((extra, 3)) - 0.5)]))
    fvel = f32(np.concatenate([fvel, rng.normal(size=(extra, 3))]))
    st = system.make_star(4, 3, 0.5, 5.0, 1.0, np.random.default_rng(5), bond=0.97)
    spec = system.ReplicaSpec(L=L, arms=4, n_arm=3, solvophobic_fraction=0.5, shear=0.2, seed=77)
    reps = [dict(W.replica_desc(spec, st), n_fluid=len(fpos))]
    reps += [dict(L=(b,) * 3, n_fluid=0, n_mono=0, kT=1.0, shear=0.0, h=W.H, seed=1) for b in beside]
    with capi.Context(reps, precision=capi.FP32, rng=capi.RNG_PHILOX, mono_bin=capi.MONOBIN_WRAPPED,
                      delrx_mode=capi.DELRX_PHYSICAL, step_update=W.N_SUB, max_neighbors=W.MAX_NB,
                      strict_cells=0) as ctx:
        ctx.set_fluid(0, fpos, fvel)
        ctx.set_monomers(0, f32(st.pos), f32(st.vel), np.zeros_like(st.pos), np.full(st.n, st.mass), st.amphi,
                         st.anchor)
        ctx.set_bonds(0, st.bond_src, st.bond_dst)
        ctx.init_md()
        ctx.cycles(cycles)
        ctx.raise_on_device_error()
        return ctx.get_fluid(0) + ctx.get_monomers(0)


@pytest.mark.parametrize("extra", [0, 250])
def test_results_do_not_depend_on_the_tiles(extra):
    want = _run((), extra)
    for beside in ((20,), (40,)):
        for a, b in zip(_run(beside, extra), want):
            np.testing.assert_array_equal(a, b)
