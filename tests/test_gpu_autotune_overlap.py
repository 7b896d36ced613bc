"""One periodic box runs its binning beside its MD, so the autotuner times whole
captured cycles there; two boxes run in order, and it times the phases."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi, system, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rep", [1, 2])
def test_autotuner_times_the_cycle_that_runs(n_rep):
    L, n_stars = 30, 2
    sol = system.star_solution(n_stars, 5, 11, 0.5, 5.0, 1.0, (L,) * 3, np.random.default_rng(17), bond=0.97,
                               outward_bias=0.15)
    spec = system.ReplicaSpec(L=L, arms=5, n_arm=11, solvophobic_fraction=0.5, shear=0.1, seed=23, n_stars=n_stars)
    with capi.Context([W.solution_desc(spec, sol)] * n_rep, precision=capi.FP32, rng=capi.RNG_PHILOX,
                      mono_bin=capi.MONOBIN_WRAPPED, delrx_mode=capi.DELRX_PHYSICAL, step_update=W.N_SUB,
                      max_neighbors=W.MAX_NB, strict_cells=0) as ctx:
        for k in range(n_rep):
            ctx.init_solvent(k, seed=3 + k, shear_profile=True)
            ctx.set_monomers(k, sol.pos, sol.vel, np.zeros_like(sol.pos), np.full(sol.n, 5.0), sol.amphi, sol.anchor)
            ctx.set_bonds(k, sol.bond_src, sol.bond_dst)
        ctx.init_md()
        ctx.cycles(3)
        before = ctx.get_fluid(0) + ctx.get_monomers(0)
        report = ctx.autotune(4)
        chosen = ctx.get_variants()[0], ctx.get_pmd_variant()
        assert chosen == (report["fluid_bin"]["index"], report["pmd"]["index"])
        for a, b in zip(before, ctx.get_fluid(0) + ctx.get_monomers(0)):
            np.testing.assert_array_equal(a, b)
        ms = list(report["fluid_bin"]["ms_per_cycle"].values())
        md = min(report["pmd"]["ms_per_cycle"].values())
        # a cycle holds ten substeps of two launches each, the binning is one launch
        assert (min(ms) > 0.5 * md) if n_rep == 1 else (max(ms) < 0.5 * md)
        ctx.cycles(2)
        ctx.raise_on_device_error()
