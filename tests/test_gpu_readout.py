"""Output-step sums against numpy where their rules can go wrong: profile bins
at exact multiples of the width and at the faces, runs of slots in any order,
boxes smaller than one block's slots, and the pressure tensor of a fluid."""
import numpy as np
import pytest

from starpolymersmd_gb300 import capi

pytestmark = pytest.mark.gpu


def _round(x):  # half away from zero, as round() of the reference
    return np.sign(x) * np.floor(np.abs(x) + 0.5)


def _profile(pos, vel, L, shear, delrx, width):
    x, v = pos.copy(), vel.copy()
    if shear:
        cy = _round(x[:, 1] / L[1])
        x[:, 0] -= L[0] * _round(x[:, 0] / L[0])
        x[:, 0] -= cy * delrx
        x[:, 0] -= L[0] * _round(x[:, 0] / L[0])
        x[:, 1] -= L[1] * cy
        v[:, 0] -= cy * shear * L[1]
    else:
        x -= _round(x / np.asarray(L, float)) * np.asarray(L, float)
    out = []
    for a in range(2):
        k0 = int(np.floor(-L[a] / (2.0 * width)))
        n = int(np.floor(L[a] / (2.0 * width))) - k0 + 1
        k = np.floor(x[:, a] / width).astype(int) - k0
        ok = (k >= 0) & (k < n)
        out.append(np.stack([np.bincount(k[ok], w[ok], n) for w in (v[:, 0], v[:, 1], np.ones(len(k)))],
                            axis=1))
    return out


@pytest.mark.parametrize("precision", [capi.FP32, capi.FP64])
@pytest.mark.parametrize("L,n_c,width,shear", [((5, 6, 7), 1, 1.0, 0.1), ((11, 9, 8), 10, 0.25, 0.0),
                                               ((12, 7, 10), 10, 0.3, 0.2), ((16, 16, 16), 3, 7.5, 0.05),
                                               ((9, 9, 9), 4, 40.0, 0.1)])
def test_velocity_profile_bins(precision, L, n_c, width, shear):
    rng = np.random.default_rng(int(100 * width) + L[0])
    n = n_c * int(np.prod(L))
    pos = (rng.random((n, 3)) - 0.5) * np.asarray(L, float)
    # every fourth particle on a multiple of the width, some at the faces and
    # at the origin, some past the faces by up to a box length
    pos[::4, 0] = np.round(pos[::4, 0] / width) * width
    pos[1::4, 1] = np.round(pos[1::4, 1] / width) * width
    pos[0] = [L[0] / 2, -L[1] / 2, 0.0]
    pos[1] = [-L[0] / 2, L[1] / 2, 0.0]
    pos[2:6, :2] = [[0.0, 0.0], [L[0] * 0.9, 0.0], [0.0, L[1] * 1.2], [-L[0] * 1.4, -L[1] * 0.6]]
    vel = rng.normal(size=(n, 3))
    vel[7] = 0.0
    if precision == capi.FP32:
        pos, vel = (a.astype(np.float32).astype(np.float64) for a in (pos, vel))
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=shear, h=0.1, seed=3)], precision=precision,
                      rng=capi.RNG_PHILOX, step_update=1, strict_cells=0) as ctx:
        ctx.set_fluid(0, pos, vel)
        ctx.set_delrx(0, 0.7)
        for cycles in (0, 2):  # slots in id order, then in cell order
            if cycles:
                ctx.set_fluid(0, (rng.random((n, 3)) - 0.5) * np.asarray(L, float), vel)
                ctx.cycles(cycles)
                ctx.raise_on_device_error()
                pos, vel = ctx.get_fluid(0)
            got = ctx.velocity_profile(0, width)
            want = _profile(pos, vel, L, shear, ctx.delrx(0), width)
            for g, w in zip(got, want):
                np.testing.assert_array_equal(g[:, 2], w[:, 2])
                # sums of up to n terms of size ~5: n eps times that
                np.testing.assert_allclose(g[:, :2], w[:, :2], rtol=0, atol=n * 5 * 2.3e-16 * 4)


@pytest.mark.parametrize("precision", [capi.FP32, capi.FP64])
@pytest.mark.parametrize("mass", [1.0, 2.5])
def test_kinetic_tensor_of_a_fluid(precision, mass):
    rng = np.random.default_rng(5)
    L, n, shear = (13, 7, 9), 8000, 0.3
    pos = (rng.random((n, 3)) - 0.5) * np.asarray(L, float)
    vel = rng.normal(size=(n, 3))
    vel[3], pos[4], vel[5, 1] = 0.0, 0.0, 1e-40  # zeros and a float32 subnormal
    if precision == capi.FP32:
        pos, vel = (a.astype(np.float32).astype(np.float64) for a in (pos, vel))
    with capi.Context([dict(L=L, n_fluid=n, kT=1.0, shear=shear, h=0.1, seed=3, solvent_mass=mass)],
                      precision=precision, rng=capi.RNG_PHILOX, step_update=1, strict_cells=0) as ctx:
        ctx.set_fluid(0, pos, vel)
        kin, vir = ctx.pressure_tensor_all()
    u = vel - shear * pos[:, 1:2] * np.array([1.0, 0.0, 0.0])
    P = mass * (u.T @ u) / np.prod(L)
    want = P[[0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2]]
    # n terms of size ~10 over the volume, rounded n times at the most
    np.testing.assert_allclose(kin[0], want, rtol=0, atol=n * 10 * mass / np.prod(L) * n * 2.3e-16)
    assert not vir.any()
