"""FP32 substeps with the Verlet lists in shared memory (launch shapes 0, 2 and 3)
against the kernel that reads them from global memory (shape 1): bead counts on
both sides of each number of lanes per bead, lists and bonds that outgrow the
shared memory, lists of an earlier call, both potentials and both thermostats.

Both sides follow the FP64 oracle to 1e-4 in the positions and 2e-3 of the
largest velocity, force and energy over 20 substeps (the bounds of the launch
shapes' own test), so they lie within twice that of each other."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi, system, workloads as W

pytestmark = pytest.mark.gpu

# arms, beads per arm, r_verlet, copies of every bond, potential, Andersen
LJ, REF = capi.POT_LJ126, capi.POT_REF4824
CASES = {
    "2": (1, 1, 3.0, 1, LJ, False),
    "64": (7, 9, 3.0, 1, LJ, False),
    "65": (8, 8, 3.0, 1, REF, False),
    "128": (1, 127, 3.0, 1, LJ, True),
    "129": (8, 16, 3.0, 1, LJ, False),
    "256": (5, 51, 3.0, 1, REF, True),
    "257": (16, 16, 3.0, 1, LJ, False),
    "512": (7, 73, 3.0, 1, LJ, False),
    "513": (16, 32, 3.0, 1, LJ, True),
    "1024": (11, 93, 3.0, 1, LJ, False),
    "lists_outgrow": (12, 30, 9.0, 1, LJ, False),
    "bonds_outgrow": (8, 50, 3.0, 2, LJ, False),
}


def _run(case, variant, large=True):
    arms, n_arm, r_verlet, copies, pot, andersen = CASES[case]
    specs = [system.ReplicaSpec(L=40, arms=arms, n_arm=n_arm, solvophobic_fraction=0.6, shear=0.1,
                                seed=71),
             system.ReplicaSpec(L=40, arms=13, n_arm=40, solvophobic_fraction=0.4, shear=0.1,
                                seed=72)]
    stars, descs = [], []
    for s in specs if large else specs[:1]:
        st = system.make_star(s.arms, s.n_arm, s.solvophobic_fraction, s.mono_mass, s.kT,
                              np.random.default_rng(300 + s.seed), bond=0.97)
        stars.append(st)
        d = W.replica_desc(s, st)
        d["potential"] = pot
        if pot == REF:
            d["r_cut"], d["r_verlet"] = 1.5, 2.0
        else:
            d["r_verlet"] = r_verlet
        descs.append(d)
    kw = dict(md_thermostat=capi.MDTHERMO_ANDERSEN, andersen_nu=1.0) if andersen else {}
    with capi.Context(descs, precision=capi.FP32, rng=capi.RNG_PHILOX, max_neighbors=1024,
                      step_update=W.N_SUB, strict_cells=0, **kw) as ctx:
        ctx.set_variants(0, 0, variant)
        for k, st in enumerate(stars):
            ctx.set_monomers(k, st.pos, st.vel, np.zeros_like(st.pos), np.full(st.n, st.mass),
                             st.amphi, st.anchor)
            ctx.set_bonds(k, np.repeat(st.bond_src, copies), np.repeat(st.bond_dst, copies))
        ctx.init_md()
        for n in (1, 3, 1, 10, 4):  # most calls begin with the lists of the one before
            ctx.md_substeps(n)
        ctx.md_substeps(1, calc_epot=True)
        ctx.raise_on_device_error()
        return [ctx.get_monomers(k) + (np.array(ctx.epot(k)),) for k in range(len(stars))]


@pytest.mark.parametrize("case", list(CASES))
def test_lists_in_shared_memory_match_those_in_global_memory(case):
    want = _run(case, 1)
    # shape 0 without the second star, of more than 512 beads, runs 512 threads
    for variant, large in ((0, True), (0, False), (2, True), (3, True)):
        for got, ref in zip(_run(case, variant, large), want):
            np.testing.assert_allclose(got[0], ref[0], rtol=0, atol=2e-4)
            for g, r in zip(got[1:], ref[1:]):
                np.testing.assert_allclose(g, r, rtol=0, atol=4e-3 * np.abs(r).max())
