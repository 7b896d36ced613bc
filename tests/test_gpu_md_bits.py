"""The FP32 substeps with lists in shared memory (launch shape 0) and those with the
lists in global memory (shape 1), both with one lane per bead, give the same bits:
the Verlet lists, their order and the order of every sum are the same, and the pairs
that shape 0 leaves out of its own lists carry exactly zero force until the next
rebuild."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi, system, workloads as W

pytestmark = pytest.mark.gpu

# arms, beads per arm, solvophobic share, r_cut, r_verlet, potential, Andersen
LJ, REF = capi.POT_LJ126, capi.POT_REF4824
CASES = {
    "121": (6, 20, 0.5, 2.5, 2.8, LJ, False),
    "401": (10, 40, 0.5, 2.5, 2.8, LJ, True),
    "513": (16, 32, 0.6, 2.5, 2.8, LJ, False),
    "1024": (11, 93, 0.4, 2.5, 3.0, LJ, False),
    "reference_potential": (8, 30, 0.5, 1.5, 2.0, REF, False),
    "thin_skin": (6, 30, 0.5, 2.5, 2.55, LJ, False),
    # r_verlet below r_cut: the displacement that asks for a rebuild is |r_verlet - r_cut| / 2
    "repulsive_below_r_cut": (8, 40, 0.0, 2.5, 1.6, LJ, False),
    "reference_below_r_cut": (8, 40, 0.0, 1.5, 1.1, REF, True),
    "attracting_below_r_cut": (8, 40, 0.5, 4.0, 2.8, LJ, False),
}


def _run(case, shape, calls):
    """State after init_md and after every call, n substeps or (n, whether the energy is reported)."""
    arms, n_arm, frac, r_cut, r_verlet, pot, andersen = case
    spec = system.ReplicaSpec(L=40, arms=arms, n_arm=n_arm, solvophobic_fraction=frac, shear=0.1, seed=71)
    st = system.make_star(arms, n_arm, frac, spec.mono_mass, spec.kT, np.random.default_rng(371), bond=0.97)
    desc = dict(W.replica_desc(spec, st), n_fluid=0, potential=pot, r_cut=r_cut, r_verlet=r_verlet)
    kw = dict(md_thermostat=capi.MDTHERMO_ANDERSEN, andersen_nu=1.0) if andersen else {}
    out = []
    with capi.Context([desc], precision=capi.FP32, rng=capi.RNG_PHILOX, max_neighbors=1024,
                      step_update=W.N_SUB, strict_cells=0, **kw) as ctx:
        ctx.set_variants(0, 0, shape)
        ctx.set_monomers(0, st.pos, st.vel, np.zeros_like(st.pos), np.full(st.n, st.mass), st.amphi, st.anchor)
        ctx.set_bonds(0, st.bond_src, st.bond_dst)
        ctx.init_md()
        out.append(ctx.get_monomers(0))
        for n in calls:  # most calls begin with the lists of the one before
            n, epot = n if isinstance(n, tuple) else (n, False)
            ctx.md_substeps(n, calc_epot=epot)
            out.append(ctx.get_monomers(0) + ((ctx.epot(0),) if epot else ()))
        if pot == LJ:  # (the reference's FENE reports bonds that a random start overstretches)
            ctx.raise_on_device_error()
        return out, ctx.verlet_rebuilds(0)


@pytest.mark.parametrize("case", list(CASES))
def test_lists_in_shared_memory_give_the_same_bits(case):
    calls = (1, 3, 1, 10, 25)
    (got, rebuilds), (want, expected) = (_run(CASES[case], shape, calls) for shape in (0, 1))
    assert rebuilds == expected
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            np.testing.assert_array_equal(a, b)


# calls whose last substep reports the energy, from the lists of a call before (1), of
# its own first substeps (3), after a rebuild; and lists that outgrow the shared memory
@pytest.mark.parametrize("arms,n_arm,r_verlet", [(6, 20, 2.8), (10, 40, 2.8), (11, 93, 3.0), (12, 30, 9.0)])
def test_substeps_that_report_the_energy_give_the_same_bits(arms, n_arm, r_verlet):
    calls = ((1, True), (1, True), 5, (1, True), (3, True), 12, (1, True), 1)
    case = (arms, n_arm, 0.5, 2.5, r_verlet, LJ, False)
    (got, rebuilds), (want, expected) = (_run(case, shape, calls) for shape in (0, 1))
    assert rebuilds == expected
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            if np.ndim(b):
                np.testing.assert_array_equal(a, b)
            else:  # the energy: terms of some 100 in all per bead, each of a few FP32 roundings
                np.testing.assert_allclose(a, b, rtol=0, atol=100 * len(w[0]) * 4 * 2.0 ** -24)


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_forces_of_beads_far_from_the_first(sign):
    # two straight arms side by side reach 80 list cells from bead 0; beads past 64 are
    # listed in another order, so the sums of up to twenty terms below 60 round differently
    n_arm = 110
    k = np.arange(1, n_arm + 1)
    arms = [np.stack([sign * 0.97 * k, np.full(n_arm, 1.05 * a), 0.03 * np.sin(1.0 * k)], axis=1) for a in range(2)]
    pos = np.concatenate([[[0.0, 0.5, 0.0]], *arms])
    n = len(pos)
    src = np.concatenate([[0], np.arange(1, n_arm), [0], np.arange(n_arm + 1, n - 1)])
    dst = np.concatenate([[1], np.arange(2, n_arm + 1), [n_arm + 1], np.arange(n_arm + 2, n)])
    rep = dict(L=(300, 20, 20), n_fluid=0, n_mono=n, mol0_size=n, kT=1.0, shear=0.0, h=0.1, md_dt=0.01, seed=1,
               potential=LJ, r_cut=1.13, r_verlet=1.3, **{"lambda": 1.0})
    forces = []
    for shape in (0, 1, 2):
        with capi.Context([rep], precision=capi.FP32, rng=capi.RNG_PHILOX, step_update=1, strict_cells=0) as ctx:
            ctx.set_variants(0, 0, shape)
            ctx.set_monomers(0, pos, np.zeros_like(pos), np.zeros_like(pos), np.full(n, 5.0), np.zeros(n, np.int32),
                             np.zeros(n, np.int32))
            ctx.set_bonds(0, src, dst)
            ctx.init_md()
            ctx.raise_on_device_error()
            forces.append(ctx.get_monomers(0)[2])
    for f in (forces[0], forces[2]):
        np.testing.assert_allclose(f, forces[1], rtol=0, atol=20 * 2.0 ** -24 * 60)
    assert np.abs(forces[1][n_arm - 5:n_arm]).max() > 1.0
