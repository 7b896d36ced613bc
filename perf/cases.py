"""What the framework's speed is measured on: the calls that a user's program makes between two of its own steps.

Kinds of a case (``kind``):
  cycles    ``Context.cycles``: step_update MD substeps and one collision per cycle, the state staying on the GPU, then
            the device's error word, which a run looks at between its blocks of cycles
  io        ``Context.cycles_io``: monomer state in from pinned memory, the cycles, monomer state and output-step
            observables out (a host program that looks at every step)
  dropin    the reference driver's loop through the step-wise calls: one ``md_substeps`` and one ``mpc_step`` per
            iteration, every step_update-th a collision with the host's random numbers
  md        ``Context.md_substeps`` with the Andersen thermostat and no solvent (the reference's MPC-off runs)
  readout   the output step's observables: molecules, velocity profile, pressure tensor

Boxes (``box``): ``star`` one star in its own box, ``table`` many uneven boxes of one star each
(``system.batched_replica_table``), ``solution`` many stars in one periodic box, ``fluid`` solvent alone.
``shapes`` are the launch shapes that the autotuner keeps for such a workload on GB300 (a program that is tuned starts
with them from the autotuner's cache); empty: the library's own defaults.

Solvent: about ``n_c`` particles per cell, uniform, Maxwell-Boltzmann at kT = 1; stars: self-avoiding walks in a random
orientation, mass 5 beads, half of them solvophobic. The 12-6 preset with skin 0.3 and 10 substeps of 0.01 per
collision (h = 0.1), as the workloads of ``starpolymersmd_gb300.workloads``; ``dropin`` runs the reference's own 48-24
potentials and options. What an FP32 context gives (its observables too, whose sums are in 64 bits) is compared as the
float32 numbers that its state holds.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from starpolymersmd_gb300 import capi, system, workloads

N_SUB, H, MD_DT, MASS, KT = workloads.N_SUB, workloads.H, workloads.MD_DT, 5.0, 1.0
HOST_FLUID = 8_000_000  # solvent up to here comes from the host (a read-in state), above from the device's initialiser


def _case(kind, box, **kw):
    c = dict(kind=kind, box=box, L=20, Ly=0, Lz=0, arms=6, n_arm=20, n_stars=1, n_rep=1, table=1, n_c=10, shear=0.05,
             fp64=False, amc=False, steps=1, shapes="")
    assert not set(kw) - set(c)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest run people start with: one 121-bead star, 20^3 cells; launches and the MD's latency
        dict(_case("cycles", "star", steps=5), name="star_20"),
        # the reference's driver over the drop-in classes: FP64, host draws, one call per substep
        dict(_case("dropin", "star", L=24, n_arm=12, shear=0.01, fp64=True), name="dropin_24_fp64"),
        # the reference-precision run of one star of 401 beads in 50^3 cells
        dict(_case("cycles", "star", L=50, arms=10, n_arm=40, fp64=True), name="star_50_fp64"),
        # the same in FP32 with the launch shapes of its tuning
        dict(_case("cycles", "star", L=50, arms=10, n_arm=40, shapes="0,5,4,0"), name="star_50"),
        # a small parameter study: 32 uneven boxes, observables every cycle
        dict(_case("io", "table", n_rep=32, shapes="0,9,2,0"), name="table_32"),
        # the large parameter study: 256 uneven boxes, 65.8 M solvent particles
        dict(_case("io", "table", n_rep=256, shapes="0,9,2,0"), name="table_256"),
        # a semi-dilute solution: 64 interacting stars in one periodic 100^3 box
        dict(_case("cycles", "solution", L=100, arms=8, n_arm=40, n_stars=64, shear=0.1, shapes="0,9,0,0"), name="solution_100"),
        # the large periodic box: 16 stars, 200^3 cells, 80 M solvent particles
        dict(_case("cycles", "solution", L=200, arms=12, n_arm=30, n_stars=16, shapes="0,9,0,2"), name="solution_200"),
        # MPC-off run of one star in FP64 under the Andersen thermostat, 100 substeps a call
        dict(_case("md", "star", L=50, arms=10, n_arm=40, fp64=True, steps=100), name="andersen_401_fp64"),
        # the angular-momentum-conserving collision in an odd box, one star
        dict(_case("cycles", "star", L=31, amc=True), name="amc_31"),
        # solvent alone in an odd box that is no cube (the fluid test driver)
        dict(_case("cycles", "fluid", L=61, Ly=47, Lz=53), name="fluid_61_47_53"),
        # what the driver reads at an output step
        dict(_case("readout", "star", L=50, arms=10, n_arm=40), name="readout_50"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["star", "star", "star_io", "table", "table", "solution", "solution", "fluid", "fluid", "amc", "md",
                       "dropin", "readout"])
    shear = rng.choice([0.0, math.exp(rng.uniform(math.log(1e-3), math.log(0.5)))])
    arms, n_arm, fp64 = rng.randint(3, 12), rng.randint(10, 60), rng.random() < 0.3
    if what in ("star", "star_io"):
        shapes = "" if fp64 else rng.choice(["", "0,5,4,0", "0,9,2,0"])
        return _case("cycles" if what == "star" else "io", "star", L=_log(rng, 16, 64), arms=arms, n_arm=n_arm, shear=shear,
                     fp64=fp64, n_c=rng.choice([5, 10, 10, 20]), steps=rng.choice([1, 1, 2]), shapes=shapes)
    if what == "table":
        n = _log(rng, 2, 64)
        return _case("io", "table", n_rep=n, table=rng.randint(2, 10 ** 6), fp64=fp64 and n <= 8,
                     shapes="" if fp64 else rng.choice(["", "0,9,2,0"]))
    if what == "solution":
        L = _log(rng, 30, 150)
        stars = max(1, min(48, int(20544 * (L / 100) ** 3 * rng.uniform(0.2, 1.0) / (1 + arms * n_arm))))
        return _case("cycles", "solution", L=L, arms=arms, n_arm=n_arm, n_stars=stars, shear=shear, fp64=fp64 and L <= 80,
                     shapes="" if fp64 else rng.choice(["", "0,5,0,0", "0,9,0,1"]))
    if what == "fluid":
        L, Ly, Lz = (_log(rng, 13, 121) for _ in range(3))
        return _case("cycles", "fluid", L=L, Ly=Ly, Lz=Lz, n_c=rng.choice([3, 5, 10, 20]), shear=shear,
                     fp64=fp64 and L * Ly * Lz < 400_000, shapes="" if fp64 else rng.choice(["", "0,9,0,0"]))
    if what == "amc":
        return _case("cycles", "star", L=_log(rng, 17, 50), arms=arms, n_arm=min(n_arm, 30), shear=shear, fp64=fp64, amc=True)
    if what == "md":
        fp64 = rng.random() < 0.5  # FP32 trajectories part from each other after some tens of substeps
        return _case("md", "star", L=50, arms=arms, n_arm=n_arm, fp64=fp64, steps=_log(rng, 20, 200) if fp64 else _log(rng, 10, 30))
    if what == "dropin":
        return _case("dropin", "star", L=_log(rng, 20, 40), arms=rng.randint(3, 8), n_arm=rng.randint(5, 12), shear=0.01,
                     fp64=True)
    return _case("readout", "star", L=_log(rng, 16, 64), arms=arms, n_arm=n_arm, shear=shear, fp64=fp64)


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _shape(arms, n_arm, bond):
    """One star's positions about its core, in the reference's bead order."""
    for k in range(20):
        rng = np.random.default_rng([arms, n_arm, k])
        try:
            return system.saw_star(arms, n_arm, rng, bond=bond, anchor_bond=2.0, r_min=1.0, outward_bias=0.15)
        except RuntimeError:  # a trapped walk
            continue
    raise RuntimeError("no self-avoiding walk found")


@functools.lru_cache(maxsize=None)
def _solution(L, arms, n_arm, n_stars):
    for k in range(20):
        try:
            return system.star_solution(n_stars, arms, n_arm, 0.5, MASS, KT, (L,) * 3, np.random.default_rng([3001, k]),
                                        bond=0.97, outward_bias=0.15)
        except RuntimeError:  # a trapped walk
            continue
    raise RuntimeError("no room for the stars")


def _f32(a):
    return np.asarray(a, dtype=np.float32).astype(np.float64)


def _edges(c):
    return (c["L"], c["Ly"] or c["L"], c["Lz"] or c["L"])


def _boxes(c):
    """(edges, arms, beads per arm, solvophobic share, shear) of every box."""
    if c["box"] == "table":
        return [((s.L,) * 3, s.arms, s.n_arm, s.solvophobic_fraction, s.shear)
                for s in system.batched_replica_table(256, c["table"])[:c["n_rep"]]]
    return [(_edges(c), c["arms"], c["n_arm"], 0.5, c["shear"])]


def _inputs(c, seed):
    """Per box: solvent (pos, vel) or None, and its monomers; every value is a float32 number."""
    rng = np.random.default_rng([seed, 11])
    boxes, n_all = _boxes(c), 0
    if c["kind"] != "md":
        n_all = sum(c["n_c"] * math.prod(b[0]) for b in boxes)
    out = []
    for L, arms, n_arm, frac, shear in boxes:
        Lv = np.asarray(L, dtype=np.float64)
        n_f = c["n_c"] * math.prod(L) if c["kind"] != "md" else 0
        b = dict(L=L, shear=shear, n_f=n_f, fluid=None, n=0, mols=None, key=int(rng.integers(1, 1 << 62)))
        if 0 < n_all <= HOST_FLUID:
            pos = (rng.random((n_f, 3), dtype=np.float32) - np.float32(0.5)) * np.asarray(L, dtype=np.float32)
            vel = rng.standard_normal((n_f, 3), dtype=np.float32)
            vel -= vel.mean(axis=0, dtype=np.float64).astype(np.float32)
            if c["box"] == "solution":
                vel[:, 0] += np.float32(shear) * pos[:, 1]
            b["fluid"] = (pos.astype(np.float64), vel.astype(np.float64))
        if c["box"] == "solution":
            sol = _solution(L[0], arms, n_arm, c["n_stars"])
            move = rng.uniform(-0.5, 0.5, 3) * Lv
            p = np.concatenate([s.pos - Lv * np.round((s.pos[0] + move) / Lv) + move for s in sol.stars])
            v = rng.normal(scale=math.sqrt(KT / MASS), size=p.shape)
            v[:, 0] += shear * p[:, 1]
            b.update(n=sol.n, pos=_f32(p), vel=_f32(v), amphi=sol.amphi, anchor=sol.anchor, src=sol.bond_src,
                     dst=sol.bond_dst, mols=sol.mol_start)
        elif c["box"] != "fluid":
            B = int(round(frac * n_arm))
            amphi, anchor, src, dst = system.star_topology(arms, n_arm - B, B)
            q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
            p = _shape(arms, n_arm, 1.01 if c["kind"] == "dropin" else 0.97) @ q.T
            v = rng.normal(scale=math.sqrt(KT / MASS), size=p.shape)
            b.update(n=len(p), pos=_f32(p), vel=_f32(v - v.mean(axis=0)), amphi=amphi, anchor=anchor, src=src, dst=dst)
        out.append(b)
    return out


def _draws(c, boxes, seed):
    """The host's random numbers of one collision (dropin): grid shift, and per cell a gamma variate and the axis."""
    rng = np.random.default_rng([seed, 12])
    n = sum(math.prod(b["L"]) for b in boxes)
    return (rng.random(3 * len(boxes)) - 0.5, rng.gamma(1.5 * (c["n_c"] - 1), KT, n), rng.random(n), rng.random(n))


def prepare(case, seed):
    c, boxes = case, _inputs(case, seed)
    dropin, md, sol = c["kind"] == "dropin", c["kind"] == "md", c["box"] == "solution"
    reps = []
    for b in boxes:
        r = dict(L=b["L"], n_fluid=b["n_f"], n_mono=b["n"], kT=KT, shear=b["shear"], h=H, md_dt=MD_DT, seed=b["key"],
                 **{"lambda": 1.0})
        if not dropin:
            r.update(potential=capi.POT_LJ126, r_cut=workloads.R_CUT_LJ, r_verlet=workloads.R_CUT_LJ + workloads.SKIN)
        if sol:
            r.update(flags=capi.REPLICA_PERIODIC_MD, mol0_size=int(b["mols"][1]))
        reps.append(r)
    opt = dict(precision=capi.FP64 if c["fp64"] else capi.FP32, step_update=N_SUB, angular_momentum=c["amc"])
    if not dropin:  # dropin: host draws, and the options' own defaults, which are the reference's
        opt.update(rng=capi.RNG_PHILOX, mono_bin=capi.MONOBIN_WRAPPED, delrx_mode=capi.DELRX_PHYSICAL,
                   max_neighbors=workloads.MAX_NB, strict_cells=0)
    if md:
        opt.update(md_thermostat=capi.MDTHERMO_ANDERSEN, andersen_nu=5.0)
    ctx = capi.Context(reps, **opt)
    for k, b in enumerate(boxes):
        if b["fluid"] is not None:
            ctx.set_fluid(k, *b["fluid"])
        elif b["n_f"]:
            ctx.init_solvent(k, seed=b["key"], shear_profile=sol)
        if b["n"]:
            ctx.set_monomers(k, b["pos"], b["vel"], np.zeros_like(b["pos"]), np.full(b["n"], MASS), b["amphi"], b["anchor"])
            ctx.set_bonds(k, b["src"], b["dst"])
        if sol:
            ctx.set_molecules(k, b["mols"])
    ctx.init_md()
    if c["shapes"]:
        *v, pmd = (int(x) for x in c["shapes"].split(","))
        ctx.set_variants(*v)
        ctx.set_pmd_variant(pmd)
    ctx.synchronize()
    s = dict(ctx=ctx, case=dict(c), t=0, real=np.float64 if c["fp64"] else np.float32, n=[b["n"] for b in boxes],
             nf=[b["n_f"] for b in boxes])
    if c["kind"] == "io":  # the host program's own pinned arrays
        m = sum(s["n"])
        s["pos"], s["vel"] = (torch.empty((m, 3), dtype=torch.float64).pin_memory().numpy() for _ in range(2))
        s["obs"] = torch.empty((len(boxes), capi.OBS_PER_REP), dtype=torch.float64).pin_memory().numpy()
        s["pos"][:] = np.concatenate([b["pos"] for b in boxes])
        s["vel"][:] = np.concatenate([b["vel"] for b in boxes])
    if dropin:
        s["draws"] = _draws(c, boxes, seed)
    return s


# --------------------------------------------------------------------- run

class _Held(dict):
    """Outputs that the context holds on the GPU, each read back when it is looked at."""

    def __getitem__(self, key):
        return super().__getitem__(key)()


def _held(s):
    ctx, real, reps = s["ctx"], s["real"], range(len(s["n"]))

    def read(get, part, counts):
        return lambda: np.concatenate([get(k)[part].astype(real) for k in reps if counts[k]])

    out = _Held()
    if any(s["nf"]):
        out["fluid_pos"], out["fluid_vel"] = (read(ctx.get_fluid, q, s["nf"]) for q in range(2))
    if any(s["n"]):
        out["mono_pos"], out["mono_vel"], out["mono_force"] = (read(ctx.get_monomers, q, s["n"]) for q in range(3))
    return out


def run(state):
    s, ctx = state, state["ctx"]
    kind, steps = s["case"]["kind"], s["case"]["steps"]
    if kind == "cycles":
        ctx.cycles(steps)
        return {"state": _held(s), "error_word": ctx.error_word()[0]}
    if kind == "io":
        ctx.cycles_io(steps, s["pos"], s["vel"], s["pos"], s["vel"], s["obs"])
        return {"state": _held(s), "observables": s["obs"].astype(s["real"])}
    if kind == "dropin":
        for _ in range(N_SUB):
            ctx.md_substeps(1)
            ctx.mpc_step(s["t"], H, *s["draws"])
            s["t"] += 1
        return _held(s)
    if kind == "md":
        ctx.md_substeps(steps, calc_epot=True)
        return {"state": _held(s), "epot": np.array([ctx.epot()], dtype=s["real"])}
    kin, vir = ctx.pressure_tensor_all()
    return {"molecules": ctx.molecule_observables_all(), "profile": ctx.velocity_profile(0, 1.0), "kinetic": kin,
            "virial": vir}


def work(case):
    c, boxes = case, _boxes(case)
    real = 8 if c["fp64"] else 4
    beads = [(c["n_stars"] * (1 + a * n) if c["box"] != "fluid" else 0) for _, a, n, _, _ in boxes]
    cells = sum(math.prod(b[0]) for b in boxes)
    fluid = c["n_c"] * cells if c["kind"] != "md" else 0
    if c["kind"] == "readout":  # the solvent read once, the beads and their pairs
        return {"bytes": 8 * real * fluid + 8 * real * sum(beads), "flops": 30 * fluid + 500 * sum(beads)}
    sub = {"md": c["steps"], "dropin": N_SUB}.get(c["kind"], N_SUB * c["steps"])
    turns = 1 if c["kind"] == "dropin" else c["steps"] if fluid else 0
    moved = turns * (16 * real * fluid + (24 * cells if c["kind"] == "dropin" else 0)) + 24 * real * sum(beads)
    if c["kind"] == "io":
        moved += 96 * sum(beads)
    # about 100 operations per particle and collision, 30 neighbours of 20 operations per bead and substep
    return {"bytes": moved, "flops": 100 * turns * fluid + 600 * sub * sum(beads)}


# ------------------------------------------------- the results in 64 bits

def _philox(c, k, seed):
    """Philox4x32-10 words of counters (c0, c1, c2, c3), each an array or a number, under a 64-bit key."""
    M = np.uint64(0xFFFFFFFF)
    c0, c1, c2, c3 = np.broadcast_arrays(*(np.asarray(x, dtype=np.uint64) for x in c + (k,)))
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c0 * np.uint64(0xD2511F53), c2 * np.uint64(0xCD9E8D57)
        c0, c1, c2, c3 = ((p1 >> np.uint64(32)) ^ c1 ^ np.uint64(k0), p1 & M, (p0 >> np.uint64(32)) ^ c3 ^ np.uint64(k1), p0 & M)
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _uniforms(cell, step, k, seed, fp64):
    w = _philox((cell, step & 0xFFFFFFFF, step >> 32), k, seed)
    if fp64:
        return tuple((((h << np.uint64(32)) | l) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53 + 2.0 ** -54
                     for l, h in ((w[0], w[1]), (w[2], w[3])))
    return tuple((h >> np.uint64(9)).astype(np.float64) * 2.0 ** -23 + 2.0 ** -24 for h in (w[1], w[3]))


def _gamma(cell, shape, step, seed, fp64):
    """Marsaglia-Tsang gamma variates of the cells' streams."""
    d = shape - 1.0 / 3.0
    c, out, left = 1.0 / np.sqrt(9.0 * d), np.zeros(len(d)), np.arange(len(d))
    for it in range(64):
        a, b = _uniforms(cell[left], step, 1 + 2 * it, seed, fp64)
        u, _ = _uniforms(cell[left], step, 2 + 2 * it, seed, fp64)
        x = np.sqrt(-2.0 * np.log(a)) * np.cos(2.0 * np.pi * b)
        v = (1.0 + c[left] * x) ** 3
        ok = v > 0.0
        lv = np.log(np.where(ok, v, 1.0))
        ok &= (u < 1.0 - 0.0331 * x ** 4) | (np.log(u) < 0.5 * x * x + d[left] * (1.0 - v + lv))
        out[left[ok]] = (d[left] * v)[ok]
        left = left[~ok]
        if not len(left):
            break
    return out


def _le_wrap(x, v, L, shear, delrx):
    """Lees-Edwards wrap of positions and velocities in place; the y image taken."""
    cy = np.round(x[:, 1] / L[1])
    x[:, 0] -= cy * delrx
    x[:, 1] -= cy * L[1]
    x[:, 0] -= L[0] * np.round(x[:, 0] / L[0])
    x[:, 2] -= L[2] * np.round(x[:, 2] / L[2])
    v[:, 0] -= cy * shear * L[1]
    return cy


def _forces(b, x, reference):
    """Pair and bond forces on the beads of one star (no images), their energy and their virial."""
    F, e, vir = np.zeros_like(x), 0.0, np.zeros((3, 3))
    core, cut = (1.0594631, 2.25) if reference else (2.0 ** (1.0 / 3.0), 6.25)
    i, j = np.triu_indices(b["n"], 1)
    d = x[j] - x[i]
    r2 = np.einsum("ij,ij->i", d, d)
    near = r2 < cut
    i, j, d, r2 = i[near], j[near], d[near], r2[near]
    bb = (b["amphi"][i] != 0) & (b["amphi"][j] != 0)
    inner = r2 < core
    on = np.where(inner, 1.0, np.where(bb, 1.0, 0.0))
    s = r2 ** -12 if reference else r2 ** -3
    f = on * (192.0 if reference else 48.0) / r2 * s * (s - 0.5)
    off = 0.0000593 if reference else -0.016316891136
    tail = 4.0 * (s * (s - 1.0) - off) if reference else 4.0 * s * (s - 1.0) - off
    e += np.sum(np.where(inner, 4.0 * s * (s - 1.0) + 1.0 - bb, on * tail))
    si, di = np.asarray(b["src"]), np.asarray(b["dst"])
    db = x[di] - x[si]
    q2 = np.einsum("ij,ij->i", db, db)
    R2 = np.where(np.asarray(b["anchor"])[si] != 0, 20.25, 2.25)
    if not reference:
        q2 = np.minimum(q2, 0.98 * R2)
    g = -30.0 / (1.0 - q2 / R2)
    e += np.sum(-15.0 * R2 * np.log(1.0 - q2 / R2))
    for p, q, w, m in ((i, j, d, f), (si, di, db, g)):
        t = w * m[:, None]
        for k in range(3):
            F[:, k] += np.bincount(q, t[:, k], b["n"]) - np.bincount(p, t[:, k], b["n"])
        vir += w.T @ t
    return F, e, vir


def _md(b, x, v, F, n, reference, andersen=None):
    e = 0.0
    for s in range(n):
        v += F * (0.5 * MD_DT / MASS)
        x += v * MD_DT
        F, e, _ = _forces(b, x, reference)
        v += F * (0.5 * MD_DT / MASS)
        if andersen is not None:
            nu, fp64 = andersen
            cell = np.arange(b["n"], dtype=np.uint64) | np.uint64(0x80000000)
            u = [_uniforms(cell, s, k, b["key"], fp64) for k in range(3)]
            hit = u[0][0] < nu * MD_DT
            r1, r2 = np.sqrt(-2.0 * np.log(u[0][1])), np.sqrt(-2.0 * np.log(u[1][1]))
            p1, p2 = 2.0 * np.pi * u[1][0], 2.0 * np.pi * u[2][0]
            w = math.sqrt(KT / MASS) * np.stack([r1 * np.cos(p1), r1 * np.sin(p1), r2 * np.cos(p2)], axis=1)
            v[hit] = w[hit]
    return x, v, F, e


def _collide(c, b, fx, fv, mx, mv, delrx, step, draws):
    """One collision of a box (MPC::step): recentring, streaming, sorting on the shifted grid, thermostat and rotation."""
    L, shear = np.asarray(b["L"], dtype=np.float64), b["shear"]
    n, nf = b["n"], b["n_f"]
    if n and np.any(np.abs(mx) >= 0.5 * L - 0.5):
        com, comv = mx.mean(axis=0), mv.mean(axis=0)
        mx, mv, fx, fv = mx - com, mv - comv, fx - com, fv - comv
        if shear:
            _le_wrap(fx, fv, L, shear, delrx)
    fx = fx + fv * H
    fv = fv.copy()
    _le_wrap(fx, fv, L, shear, delrx)
    if draws is None:
        a, z = _uniforms(0xFFFFFFFF, step, 0, b["key"], True), _uniforms(0xFFFFFFFF, step, 1, b["key"], True)
        shift = np.array([a[0], a[1], z[0]]) - 0.5
    else:
        shift = np.asarray(draws[0])
    fx += shift
    _le_wrap(fx, fv, L, shear, delrx)
    sx, sv = mx + shift, mv.copy()
    if c["kind"] != "dropin":
        _le_wrap(sx, sv, L, shear, delrx)
    jump = sv - mv
    X, V = np.concatenate([fx, sx]), np.concatenate([fv, sv])
    m = np.concatenate([np.ones(nf), np.full(n, MASS)])
    Li = np.asarray(b["L"])
    q = np.clip(np.floor(X + 0.5 * L).astype(np.int64), 0, Li - 1)
    cell = q[:, 0] + Li[0] * (q[:, 1] + Li[1] * q[:, 2])
    nc = int(np.prod(Li))
    cells = np.arange(nc, dtype=np.uint64)

    def total(w):
        return np.bincount(cell, w, nc)

    cnt, mt = np.bincount(cell, minlength=nc), np.maximum(total(m), 1e-300)
    cm = np.stack([total(m * V[:, k]) / mt for k in range(3)], axis=1)
    U = V - cm[cell]
    ekin = 0.5 * total(m * np.einsum("ij,ij->i", U, U))
    if draws is None:
        g = np.zeros(nc)
        two = cnt >= 2
        g[two] = KT * _gamma(cells[two], 1.5 * (cnt[two] - 1.0), step, b["key"], c["fp64"])
        uphi, uth = _uniforms(cells, step, 0, b["key"], c["fp64"])
    else:
        g, uphi, uth = draws[1:]
    sc = np.where((cnt >= 2) & (ekin > 0.0), np.sqrt(g / np.where(ekin > 0.0, ekin, 1.0)), 1.0)
    th = 2.0 * (uth - 0.5)
    st = np.sqrt(1.0 - th * th)
    a = np.stack([st * np.cos(2.0 * np.pi * uphi), st * np.sin(2.0 * np.pi * uphi), th], axis=1)
    ca, sa = math.cos(math.radians(130.0)), math.sin(math.radians(130.0))
    U *= sc[cell][:, None]
    ax = a[cell]
    W = ca * U + sa * np.cross(ax, U) + (1.0 - ca) * ax * np.einsum("ij,ij->i", ax, U)[:, None]
    V = cm[cell] + W
    if c["amc"]:
        cp = np.stack([total(m * X[:, k]) / mt for k in range(3)], axis=1)
        r = X - cp[cell]
        lost = np.cross(r, U - W) * m[:, None]
        lost = np.stack([total(lost[:, k]) for k in range(3)], axis=1)
        I = np.empty((nc, 3, 3))
        r2 = np.einsum("ij,ij->i", r, r)
        for k in range(3):
            for l in range(3):
                I[:, k, l] = total(m * ((r2 if k == l else 0.0) - r[:, k] * r[:, l]))
        use, w = cnt > 2, np.zeros((nc, 3))
        w[use] = np.linalg.solve(I[use], lost[use][:, :, None])[:, :, 0]
        V += np.cross(w[cell], r)
    fx, fv = X[:nf] - shift, V[:nf]
    _le_wrap(fx, fv, L, shear, delrx)
    return fx, fv, mx, V[nf:] - jump


def _observables(b, x, v):
    r, u = x - x.mean(axis=0), v - v.mean(axis=0)
    G, S = r.T @ r / b["n"], r.T @ r
    om = np.linalg.solve(np.trace(S) * np.eye(3) - S, np.cross(r, u).sum(axis=0))
    e = 0.5 * MASS * np.sum(u * u)
    return np.concatenate([[math.sqrt(np.trace(G))], G.ravel(), om, [e, 2.0 * e / (3.0 * (b["n"] - 1.0)), 1.0]])


def _readout(c, b):
    fx, fv = (a.copy() for a in b["fluid"])
    L, shear, x, v = np.asarray(b["L"], dtype=np.float64), b["shear"], b["pos"], b["vel"]
    flow = np.array([shear, 0.0, 0.0])
    P = np.zeros((3, 3))
    for m, q, u in ((1.0, fx, fv), (MASS, x, v)):
        w = u - q[:, 1:2] * flow
        P += m * (w.T @ w)
    vol, six = np.prod(L), ([0, 1, 2, 0, 0, 1], [0, 1, 2, 1, 2, 2])
    vir = _forces(b, x, False)[2]
    fx -= x.mean(axis=0)
    fv -= v.mean(axis=0)
    _le_wrap(fx, fv, L, shear, 0.0)
    prof = []
    for a in range(2):
        k0 = math.floor(-b["L"][a] / 2.0)
        n = math.floor(b["L"][a] / 2.0) - k0 + 1
        k = np.floor(fx[:, a]).astype(np.int64) - k0
        prof.append(np.stack([np.bincount(k, fv[:, 0], n), np.bincount(k, fv[:, 1], n), np.bincount(k, minlength=n)], axis=1))
    return {"molecules": _observables(b, x, v)[None], "profile": tuple(prof), "kinetic": (P[six] / vol)[None],
            "virial": (vir[six] / vol)[None]}


def exact(case, seed):
    """The first pass's outputs in 64 bits; None where the boxes hold more than the solvent that a host reads in (the
    device draws those states) and for interacting stars in a periodic box, both of which take too long here."""
    c = case
    if c["box"] == "solution":
        return None
    boxes = _inputs(c, seed)
    if c["kind"] == "readout":
        return _readout(c, boxes[0])
    if c["kind"] != "md" and any(b["fluid"] is None for b in boxes):
        return None
    reference = c["kind"] == "dropin"
    draws = _draws(c, boxes, seed) if reference else None
    got = {k: [] for k in ("fluid_pos", "fluid_vel", "mono_pos", "mono_vel", "mono_force")}
    obs, epot = [], 0.0
    for b in boxes:
        x, v = (b["pos"].copy(), b["vel"].copy()) if b["n"] else (np.zeros((0, 3)), np.zeros((0, 3)))
        F = _forces(b, x, reference)[0] if b["n"] else x
        if c["kind"] == "md":
            x, v, F, epot = _md(b, x, v, F, c["steps"], False, (5.0, c["fp64"]))
        else:
            fx, fv, delrx = b["fluid"][0].copy(), b["fluid"][1].copy(), 0.0
            adv = b["shear"] * b["L"][1] * H / (1.0 if reference else N_SUB)
            for step in range(c["steps"]):
                for k in range(N_SUB if reference else 1):  # the driver's loop collides in its first iteration
                    if b["n"]:
                        x, v, F, _ = _md(b, x, v, F, 1 if reference else N_SUB, reference)
                    delrx += adv * (1 if reference else N_SUB)
                    delrx -= b["L"][0] * round(delrx / b["L"][0])
                    if k == 0:
                        fx, fv, x, v = _collide(c, b, fx, fv, x, v, delrx, step, draws)
            got["fluid_pos"].append(fx)
            got["fluid_vel"].append(fv)
        if b["n"]:
            got["mono_pos"].append(x)
            got["mono_vel"].append(v)
            got["mono_force"].append(F)
            if c["kind"] == "io":
                obs.append(_observables(b, x, v))
    got = {k: np.concatenate(p) for k, p in got.items() if p}
    if c["kind"] == "io":
        return {"state": got, "observables": np.stack(obs)}
    if c["kind"] == "md":
        return {"state": got, "epot": np.array([epot])}
    return got if reference else {"state": got}
