"""One periodic box bins its solvent beside its MD substeps; with a second box in the
context everything runs in order. The first box comes out the same either way."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi, system, workloads as W

pytestmark = pytest.mark.gpu


def _cycles(precision, n_rep, n_stars, shear, cycles):
    L, arms, n_arm = 40, 5, 11
    rng = np.random.default_rng(17)
    sol = system.star_solution(n_stars, arms, n_arm, 0.5, 5.0, 1.0, (L,) * 3, rng, bond=0.97,
                               outward_bias=0.15)
    spec = system.ReplicaSpec(L=L, arms=arms, n_arm=n_arm, solvophobic_fraction=0.5, shear=shear, seed=23,
                              n_stars=n_stars)
    n = 10 * L ** 3
    fpos = ((rng.random((n, 3)) - 0.5) * L).astype(np.float32).astype(float)
    fvel = rng.normal(size=(n, 3)).astype(np.float32).astype(float)
    pos, vel = sol.pos.astype(np.float32).astype(float), sol.vel.astype(np.float32).astype(float)
    desc = W.solution_desc(spec, sol)
    with capi.Context([desc] * n_rep, precision=precision, rng=capi.RNG_PHILOX, mono_bin=capi.MONOBIN_WRAPPED,
                      delrx_mode=capi.DELRX_PHYSICAL, step_update=W.N_SUB, max_neighbors=W.MAX_NB,
                      strict_cells=0) as ctx:
        for k in range(n_rep):
            ctx.set_fluid(k, fpos, fvel)
            ctx.set_monomers(k, pos, vel, np.zeros_like(pos), np.full(sol.n, 5.0), sol.amphi, sol.anchor)
            ctx.set_bonds(k, sol.bond_src, sol.bond_dst)
        ctx.init_md()
        ctx.cycles(cycles)
        ctx.raise_on_device_error()
        return ctx.get_fluid(0) + ctx.get_monomers(0) + (np.array(ctx.delrx(0)),)


# 56 and 1,120 beads: the monomers in one block and in two
@pytest.mark.parametrize("precision", [capi.FP32, capi.FP64], ids=["fp32", "fp64"])
@pytest.mark.parametrize("n_stars,shear", [(1, 0.0), (20, 0.3)])
def test_binning_beside_the_md_gives_the_cycle_in_order(precision, n_stars, shear):
    alone = _cycles(precision, 1, n_stars, shear, 3)
    pair = _cycles(precision, 2, n_stars, shear, 3)
    for a, b in zip(alone, pair):
        if precision == capi.FP32:  # sums over a cell do not depend on the order of its particles
            np.testing.assert_array_equal(a, b)
        else:  # they do in FP64, by its round-off over three collisions
            np.testing.assert_allclose(a, b, rtol=0, atol=1e-11 * max(1.0, np.abs(b).max()))
