"""FP64 cell indices where they do not come from the coordinate's bits: coordinates of
2^20 and more, and strict cells left of and beyond the box, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc
from starpolymersmd_gb300 import capi, system
from tests import gpu_helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strict", [0, 1])
def test_cells_past_two_to_the_twentieth(strict):
    L = (1, 1, 1_060_000)  # 2^20 = 1,048,576
    rng = np.random.default_rng(8)
    n = 200_000
    fpos = (rng.random((n, 3)) - 0.5) * np.array(L)
    fpos[: n // 2, 2] = L[2] / 2 - 12_000 + 11_900 * rng.random(n // 2)  # half of them around 2^20
    fvel = rng.normal(size=(n, 3))
    n_cell = L[2]
    inj = (np.array([0.3, -0.2, 0.1]), rng.gamma(13.5, 1.0, n_cell), rng.random(n_cell), rng.random(n_cell))
    o = orc.OracleSystem(L, 1.0, 0.0, 1, n)
    o.set_fluid(fpos, fvel)
    o.set_inject(*inj)
    o.mpc_step(0, 0.1)
    assert o.error() == 0
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=0.0, h=0.1)], precision=capi.FP64, rng=capi.RNG_INJECT,
                      step_update=1, strict_cells=strict) as ctx:
        ctx.set_fluid(0, fpos, fvel)
        ctx.mpc_step(0, 0.1, *inj)
        ctx.raise_on_device_error()
        got, _ = ctx.cell_members(0)
        want, _ = o.cell_members()
        np.testing.assert_array_equal(got, want)
        assert (want >= 1 << 20).sum() > 40_000
        H.close64(ctx.get_fluid(0)[1], o.get_fluid()[1])


# a third bead, apart from molecule 0, by its position after the recentring: within a
# cell left of the box and beyond it (rows run into each other), more than a cell left
# of it, and before the first and past the last cell (an error in both)
@pytest.mark.parametrize("bead,ok", [((-4.3, 0.2, 0.2), True), ((4.3, 0.2, 0.2), True), ((-5.4, 0.2, 0.2), True),
                                     ((0.2, 0.2, -4.4), True), ((0.2, 0.2, -6.4), False), ((0.2, 0.2, 4.6), False)])
def test_strict_cells_outside_the_box(bead, ok):
    L = 8
    rng = np.random.default_rng(5)
    fpos, fvel = system.uniform_fluid((L,) * 3, 10, 1.0, rng, reference_velocities=True)
    com = np.array([0.485, 0.0, 0.0])
    mpos = np.array([[0.0, 0.0, 0.0], [0.97, 0.0, 0.0], np.array(bead) + com])
    n_cell = L ** 3
    inj = (np.zeros(3), rng.gamma(13.5, 1.0, n_cell), rng.random(n_cell), rng.random(n_cell))
    o = orc.OracleSystem((L,) * 3, 1.0, 0.0, 1, len(fpos), 3, mol_start=[0, 2, 3])
    o.set_fluid(fpos, fvel)
    o.set_monomers(mpos, np.zeros((3, 3)), np.zeros((3, 3)), np.full(3, 5.0), np.zeros(3, np.int32),
                   np.zeros(3, np.int32))
    o.set_inject(*inj)
    o.mpc_step(0, 0.1)
    rep = dict(L=(L,) * 3, n_fluid=len(fpos), n_mono=3, mol0_size=2, kT=1.0, shear=0.0, h=0.1, md_dt=0.01)
    with capi.Context([rep], precision=capi.FP64, rng=capi.RNG_INJECT, step_update=1,
                      mono_bin=capi.MONOBIN_REFERENCE, strict_cells=1) as ctx:
        ctx.set_fluid(0, fpos, fvel)
        ctx.set_monomers(0, mpos, np.zeros((3, 3)), np.zeros((3, 3)), np.full(3, 5.0), np.zeros(3, np.int32),
                         np.zeros(3, np.int32))
        ctx.mpc_step(0, 0.1, *inj)
        word, info = ctx.error_word()
        assert (o.error() == 0) == ok
        if ok:
            assert word == 0
            for got, want in zip(ctx.cell_members(0), o.cell_members()):
                np.testing.assert_array_equal(got, want)
        else:
            assert word & 2 and list(info) == [2, 0, 2]
