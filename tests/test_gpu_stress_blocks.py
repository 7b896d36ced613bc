"""The pressure tensor's monomer part with its blocks dealt out over many replicas (more
than 1,216 blocks of eight beads in all): every replica's tensor is the one it has in a
context of its own, to the round-off of its sums."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi, system, workloads as W

pytestmark = pytest.mark.gpu

# arms, beads per arm: one to 128 blocks each, and a replica without monomers
SHAPES = [(1, 1), (3, 2), None, (11, 93), (6, 20), (12, 59), (10, 40), (1, 7), (1, 8)]


def _tensors(precision, shapes):
    descs, stars = [], []
    for k, shape in shapes:
        spec = system.ReplicaSpec(L=30, arms=1, n_arm=1, solvophobic_fraction=0.5, shear=0.1, seed=k + 1)
        st = None
        if shape is not None:
            st = system.make_star(*shape, 0.5, 5.0, 1.0, np.random.default_rng(40 + k % len(SHAPES)), bond=0.97)
            descs.append(dict(W.replica_desc(spec, st), n_fluid=0))
        else:
            descs.append(dict(L=(30,) * 3, n_fluid=100, n_mono=0, kT=1.0, shear=0.1, h=0.1, seed=9))
        stars.append(st)
    with capi.Context(descs, precision=precision, rng=capi.RNG_PHILOX, max_neighbors=1024, step_update=W.N_SUB,
                      strict_cells=0) as ctx:
        for k, st in enumerate(stars):
            if st is None:
                ctx.init_solvent(k, seed=4)
            else:
                ctx.set_monomers(k, st.pos, st.vel, np.zeros_like(st.pos), np.full(st.n, st.mass), st.amphi, st.anchor)
                ctx.set_bonds(k, st.bond_src, st.bond_dst)
        ctx.init_md()
        out = ctx.pressure_tensor_all()
        ctx.raise_on_device_error()
        return out


@pytest.mark.parametrize("precision", [capi.FP32, capi.FP64], ids=["fp32", "fp64"])
def test_tensors_of_many_replicas(precision):
    table = [(k, SHAPES[k % len(SHAPES)]) for k in range(9 * len(SHAPES))]  # about 2,600 blocks' worth
    kin, vir = _tensors(precision, table)
    for q in range(len(SHAPES)):
        one_kin, one_vir = _tensors(precision, [table[q]])
        # sums of at most 1024 x 1024 terms, each below the sum of the magnitudes: n eps of it
        scale = max(1e-9, np.abs(one_kin).max() + np.abs(one_vir).max())
        for k in range(q, len(table), len(SHAPES)):
            np.testing.assert_allclose(kin[k], one_kin[0], rtol=0, atol=1e-10 * scale)
            np.testing.assert_allclose(vir[k], one_vir[0], rtol=0, atol=1e-10 * scale)
