"""Workloads of the PIC step that its performance is measured by.

Each case is what a program that uses this package does between two looks at
its results: advance a plasma some steps (and, as simulations do, record the
energies on the way and take a snapshot of the fields at the end), evaluate a
gradient through the differentiable run, or audit charge conservation.  The
sizes are those of ``0buf_b200/configs.py``, of the reference's default run
and of the tests; ``draw`` spreads them over the same ranges.

A snapshot of the FP64 form is FP64.  The FP32 form stores and advances FP32
numbers, so its snapshots, energies and gradients are kept in FP32.
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

pic = importlib.import_module("0buf_b200")

EHJ = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz", "Jx", "Jy", "Jz")
FIELD_ID = {name: i for i, name in enumerate(EHJ)}
BEAM = 2


def _case(kind, cells, ppc, precision, steps, h=(0.1, 0.1, 0.1), tau=0.02, ghosts="reference", energies=False,
          stress=False, every=0, sub=0, name=None):
    c = dict(kind=kind, nx=cells[0], ny=cells[1], nz=cells[2], ppc=ppc, precision=precision, steps=steps, hx=h[0],
             hy=h[1], hz=h[2], tau=tau, ghosts=ghosts, energies=energies, stress=stress, every=every, sub=sub)
    if name:
        c["name"] = name
    return c


# the reference's default run: 100 x 4 x 4 cells, box 1.1424 x 0.05 x 0.05, tau 0.001, thousands of particles per cell
DEFAULT_H, DEFAULT_TAU = (0.011424, 0.0125, 0.0125), 0.001


def listed():
    return [
        # configuration c0, the parity case: the smallest run, where launches and waits count
        _case("run", (32, 4, 4), 32, "fp64", 10, energies=True, name="c0_fp64"),
        # a small box whose sides are multiples of nothing, periodic ghosts, as in the tests
        _case("run", (37, 13, 21), 17, "fp32", 8, ghosts="periodic", name="ragged_fp32"),
        # the reference's default run through its own step driver: few cells, very many particles in each
        _case("compute", (100, 4, 4), 1300, "fp64", 5, h=DEFAULT_H, tau=DEFAULT_TAU, name="default_fp64"),
        _case("compute", (100, 4, 4), 1300, "fp32", 5, h=DEFAULT_H, tau=DEFAULT_TAU, name="default_fp32"),
        # configuration c1: the FP64 form at scale, energies every step
        _case("run", (256, 64, 64), 64, "fp64", 10, energies=True, name="c1_fp64"),
        # configuration c2: the headline run, energies every step, fields at the end
        _case("run", (512, 128, 128), 32, "fp32", 40, energies=True, name="c2_fp32"),
        # configuration c4: non-uniform density, hot electrons, the largest time step
        _case("run", (256, 64, 64), 64, "fp32", 20, tau=0.05, stress=True, name="c4_fp32"),
        # one evaluation of a loss and its gradient, as an optimiser makes it: the smallest (the tests'),
        # configuration c3's grid and interval of checkpoints, and the FP32 form with two levels of checkpoints
        _case("grad", (16, 8, 8), 8, "fp64", 30, every=7, name="small_grad_fp64"),
        _case("grad", (128, 32, 32), 32, "fp64", 50, every=25, name="c3_grad_fp64"),
        _case("grad", (64, 32, 32), 16, "fp32", 30, every=15, sub=5, name="grad_fp32"),
        # the charge-conservation audit of a state: density, Gauss residual, momenta, energies
        _case("audit", (128, 64, 64), 32, "fp32", 1, name="audit_fp32"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("run", "run", "run", "compute", "grad", "audit"))
    precision = rng.choice(("fp64", "fp32"))
    ghosts = rng.choice(("reference", "periodic"))
    if kind == "compute":
        cells = (log(20, 120), rng.randint(3, 8), rng.randint(3, 8))
        most = 6.0e6 if precision == "fp64" else 8.0e6
        ppc = max(1, min(log(100, 1500), int(most / 3 / (cells[0] * cells[1] * cells[2]))))
        return _case(kind, cells, ppc, precision, 5, h=DEFAULT_H, tau=DEFAULT_TAU, ghosts=ghosts)
    most = {"run": {"fp64": 4.0e7, "fp32": 1.2e8}, "grad": {"fp64": 6.0e6, "fp32": 6.0e6},
            "audit": {"fp64": 4.0e7, "fp32": 8.0e7}}[kind][precision]
    cells = (log(8, 256), log(4, 96), log(4, 96))
    if kind == "grad":
        cells = (log(8, 128), log(4, 40), log(4, 40))
    n = cells[0] * cells[1] * cells[2]
    ppc = max(1, min(log(4, 96), int(most / 3 / n)))
    if kind == "run":
        stress = precision == "fp32" and rng.random() < 0.3 and min(cells) >= 8 and ppc >= 4
        return _case(kind, cells, ppc, precision, log(5, 20), tau=0.05 if stress else 0.02, ghosts=ghosts,
                     energies=rng.random() < 0.5, stress=stress)
    if kind == "grad":
        steps = log(8, 40)
        every = rng.randint(3, steps)
        sub = rng.randint(2, every) if precision == "fp32" and every > 3 and rng.random() < 0.5 else 0
        return _case(kind, cells, ppc, precision, steps, ghosts=ghosts, every=every, sub=sub)
    return _case(kind, cells, ppc, precision, 1, ghosts=ghosts)


# ------------------------------------------------------------------ state --
def _species(case):
    return pic.configs.SPECIES_STRESS if case["stress"] else pic.configs.SPECIES_BEAM_PLASMA


def _init(sim, case, seed):
    for i, s in enumerate(_species(case)):
        if "profile" in s:
            sim.init_species_profile(i, dict(s["profile"], ppc_mean=case["ppc"]), s["drift"], s["vth"], seed * 8 + i)
        else:
            sim.init_species(i, case["ppc"], s["drift"], s["vth"], seed * 8 + i)


def _smooth_fields(case, seed):
    """E of an audited state: a few plane waves with random phases, reference layout."""
    rng = np.random.RandomState(seed % (1 << 31))
    n = [case["nx"] + 2, case["ny"] + 2, case["nz"] + 2]
    x = [np.arange(v) * (2.0 * np.pi / max(v - 2, 1)) for v in n]
    out = {}
    for name in ("Ex", "Ey", "Ez"):
        a = [0.01 * np.sin(x[d] * rng.randint(1, 4) + rng.uniform(0, 6.28)) for d in range(3)]
        out[name] = (a[0][:, None, None] + a[1][None, :, None] * np.cos(x[2])[None, None, :] + a[2][None, None, :]).ravel()
    return out


def prepare(case, seed):
    cells = (case["nx"], case["ny"], case["nz"])
    lengths = tuple(c * h for c, h in zip(cells, (case["hx"], case["hy"], case["hz"])))
    st = dict(case=case, seed=int(seed))
    if case["kind"] == "compute":
        pl = pic.Plasma(*cells, *lengths, 1.0, case["ppc"], 1.0 / 1836.0, case["tau"], precision=case["precision"],
                        ghosts=case["ghosts"], seed=int(seed))
        pl.Initialize()
        st.update(plasma=pl, sim=pl.sim)
    else:
        sim = pic.PicSimulation(cells, lengths, case["tau"], pic.configs.species_table(case["ppc"], _species(case)),
                                precision=case["precision"], ghosts=case["ghosts"])
        _init(sim, case, int(seed))
        st["sim"] = sim
        if case["kind"] == "audit":
            sim.gauss_check(set_baseline=True)  # the run's own baseline
            for name, a in _smooth_fields(case, int(seed)).items():
                sim.set_field(name, a)
    nodes = int(np.prod(st["sim"].shape))
    st["zero"] = np.zeros(nodes) if case["kind"] == "grad" else None
    if case["kind"] != "grad":  # host buffers that a program with snapshots keeps
        names = EHJ + ("rho",) if case["kind"] != "audit" else ("rho", "residual")
        st["host"] = {k: torch.empty(nodes, dtype=torch.float64, pin_memory=True) for k in names}
        if case["precision"] == "fp32" and case["kind"] != "audit":
            st["host32"] = {k: torch.empty(nodes, dtype=torch.float32) for k in names}
    return st


# -------------------------------------------------------------------- run --
def _ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _check(rc, where):
    if rc != 0:
        raise pic.PicError(rc, where)


def _snapshot(st):
    """E, H, J and the charge density through the C ABI into the program's own buffers."""
    sim, host = st["sim"], st["host"]
    for name in EHJ:
        _check(sim.lib.pic_get_field(sim.h, FIELD_ID[name], _ptr(host[name])), "pic_get_field")
    _check(sim.lib.pic_charge_density(sim.h, _ptr(host["rho"])), "pic_charge_density")
    if "host32" not in st:
        return host
    for name, a in host.items():
        st["host32"][name].copy_(a)
    return st["host32"]


def _keep(case, a):
    """numbers of the FP32 form are kept in FP32"""
    return np.asarray(a, np.float32 if case["precision"] == "fp32" else np.float64)


def run(st):
    case, sim = st["case"], st["sim"]
    kind = case["kind"]
    if kind == "run":
        e = sim.run(case["steps"], energies=case["energies"])
        out = dict(fields=_snapshot(st))
        if e is not None:
            out["energies"] = _keep(case, e)
        return out
    if kind == "compute":
        st["plasma"].Compute(case["steps"])
        hist = [w for _, w in st["plasma"].energy_history[-case["steps"]:]]
        return dict(fields=_snapshot(st), history=_keep(case, hist))
    if kind == "grad":
        # the optimiser's evaluation: the initial state, the forward run, the gradient
        _init(sim, case, st["seed"])
        for name in EHJ[:6]:
            sim.set_field(name, st["zero"])
        sim.forward(case["steps"], case["every"], case["sub"] or None)
        beam = _species(case)[BEAM]
        g = sim.backward(**_loss(case, beam))
        return dict(loss=_keep(case, [g["loss"]]), d_drift=_keep(case, g["d_drift"]), d_vth=_keep(case, [g["d_vth"]]),
                    d_p0=_keep(case, g["d_p0"]), history=_keep(case, sim.history()))
    host = st["host"]
    _check(sim.lib.pic_charge_density(sim.h, _ptr(host["rho"])), "pic_charge_density")
    _check(sim.lib.pic_gauss_residual(sim.h, _ptr(host["residual"])), "pic_gauss_residual")
    return dict(fields=host, check=sim.gauss_check(), momentum=sim.momentum(), energy=sim.energy(),
                energy_reference=sim.energy_reference())


def _loss(case, beam):
    return dict(field="Ex", window=max(1, case["steps"] // 3), species=BEAM, drift=beam["drift"], vth=beam["vth"])


# ------------------------------------------------------------------- work --
def work(case):
    """Each particle read and written once a step (FP32 form: 28 bytes, FP64 form: 52), the Yee step's E, B and J
    (72 and 120 bytes a cell), the outputs once; about 260 operations a particle-step (48 field taps, the Boris
    rotation, 12 current contributions), three times that to reverse it."""
    n = case["nx"] * case["ny"] * case["nz"]
    nodes = (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
    particles = 3 * n * case["ppc"]
    wide = 2 if case["precision"] == "fp64" else 1
    state = 52 if wide == 2 else 28
    cell = 120 if wide == 2 else 72
    step = particles * 2 * state + n * cell
    if case["kind"] in ("run", "compute"):
        flops = 260.0 * particles * case["steps"]
        snapshot = particles * (16 if wide == 1 else 28) + 10 * nodes * 4 * wide
        return dict(bytes=float(step * case["steps"] + snapshot), flops=flops)
    if case["kind"] == "grad":
        # generate and forward; recompute each step, read its state, read and write the 6 adjoint values per particle
        forward = step * case["steps"] + particles * state
        backward = case["steps"] * (step + particles * (state + 2 * 6 * 4 * wide) + n * 2 * cell)
        return dict(bytes=float(forward + backward + particles // 3 * 3 * 4 * wide),
                    flops=260.0 * 5 * particles * case["steps"])
    # density: cells and positions; momenta twice (momentum, kinetic energy); E and H; rho and G
    pos = 16 if wide == 1 else 28
    return dict(bytes=float(3 * particles * pos + 2 * particles * 12 * wide + nodes * (9 + 2) * 4 * wide + nodes * 4 * 8),
                flops=60.0 * particles)


# ------------------------------------------------------------------ exact --
# The same physics in plain torch, FP64: the seeded generator, the Yee step, the field interpolation, the
# relativistic Boris push, the charge-conserving zigzag deposit in cell units.  Gradients by autograd.
_U = np.uint64


def _mix(z):
    z = z ^ (z >> _U(30))
    z = z * _U(0xBF58476D1CE4E5B9)
    z = z ^ (z >> _U(27))
    z = z * _U(0x94D049BB133111EB)
    return z ^ (z >> _U(31))


def _uniform(seed, species, cell, slot, stream):
    with np.errstate(over="ignore"):
        h = _mix(np.array([(int(seed) + 0x9E3779B97F4A7C15) % (1 << 64)], np.uint64))
        h = _mix(h ^ (_U(species) * _U(0xD6E8FEB86659FD93)))
        h = _mix(h ^ (cell * _U(0xA0761D6478BD642F)))
        h = _mix(h ^ (slot * _U(0xE7037ED1A0B428DB)))
        h = _mix(h ^ (_U(stream) * _U(0x8EBC6AF09C88C6E3)))
    return (h >> _U(11)).astype(np.float64) * (1.0 / 9007199254740992.0)


def _particles(case, seed, dev):
    """[(cell (n, 3) int64, offset (n, 3), momentum (n, 3), m, q_m)] per species"""
    nx, ny, nz, ppc = case["nx"], case["ny"], case["nz"], case["ppc"]
    cell = np.repeat(np.arange(nx * ny * nz, dtype=np.uint64), ppc)
    slot = np.tile(np.arange(ppc, dtype=np.uint64), nx * ny * nz)
    c = torch.from_numpy(cell.astype(np.int64)).to(dev)
    ijk = torch.stack([c // (ny * nz), (c // nz) % ny, c % nz], 1)
    out = []
    for s, sp in enumerate(_species(case)):
        key = int(seed) if case["kind"] == "compute" else int(seed) * 8 + s
        off = np.stack([1e-6 + _uniform(key, s, cell, slot, a) * (1.0 - 2e-6) for a in range(3)], 1)
        p = np.tile(np.array(sp["drift"], np.float64), (cell.size, 1))
        if sp["vth"]:
            r0, a0, r1, a1 = (_uniform(key, s, cell, slot, q) for q in (8, 9, 10, 11))
            r0, r1 = np.sqrt(-2.0 * np.log(1.0 - r0)), np.sqrt(-2.0 * np.log(1.0 - r1))
            w = 6.283185307179586
            p = p + sp["vth"] * np.stack([r0 * np.cos(w * a0), r0 * np.sin(w * a0), r1 * np.cos(w * a1)], 1)
        out.append([ijk.clone(), torch.from_numpy(off).to(dev), torch.from_numpy(p).to(dev),
                    math.copysign(sp["density"] / ppc, sp["q_m"]), sp["q_m"]])
    return out


def _half_b(E, H, c):
    """the increment of H by half a step, on the reference's ranges"""
    Q = [torch.zeros_like(a) for a in H]
    Q[0][:, :-1, :-1] = 0.5 * (c[2] * (E[1][:, :-1, 1:] - E[1][:, :-1, :-1]) - c[1] * (E[2][:, 1:, :-1] - E[2][:, :-1, :-1]))
    Q[1][:-1, :, :-1] = 0.5 * (c[0] * (E[2][1:, :, :-1] - E[2][:-1, :, :-1]) - c[2] * (E[0][:-1, :, 1:] - E[0][:-1, :, :-1]))
    Q[2][:-1, :-1, :] = 0.5 * (c[1] * (E[0][:-1, 1:, :] - E[0][:-1, :-1, :]) - c[0] * (E[1][1:, :-1, :] - E[1][:-1, :-1, :]))
    return Q


def _fold(J):
    out = []
    for comp in range(3):
        a = J[comp]
        for d in range(3):
            a = a.clone()
            v = a.movedim(d, 0)
            if d != comp:
                v[1] = v[1] + v[-1]
            if d != 1 or comp != 1:
                v[-1] = v[1].clone()
            v[0] = v[0] + v[-2]
            v[-2] = v[0].clone()
        out.append(a)
    return out


def _next_e(E, H, J, c, tau):
    E = [a.clone() for a in E]
    X, Y, Z = slice(0, -1), slice(1, -1), slice(0, -2)
    E[0][X, Y, Y] += c[1] * (H[2][X, Y, Y] - H[2][X, Z, Y]) - c[2] * (H[1][X, Y, Y] - H[1][X, Y, Z]) - tau * J[0][X, Y, Y]
    E[1][Y, X, Y] += c[2] * (H[0][Y, X, Y] - H[0][Y, X, Z]) - c[0] * (H[2][Y, X, Y] - H[2][Z, X, Y]) - tau * J[1][Y, X, Y]
    E[2][Y, Y, X] += c[0] * (H[1][Y, Y, X] - H[1][Z, Y, X]) - c[1] * (H[0][Y, Y, X] - H[0][Y, Z, X]) - tau * J[2][Y, Y, X]
    return E


def _ghosts(E, periodic):
    E = [a.clone() for a in E]

    def both(v):
        v[0] = v[-2].clone()
        v[-1] = v[1].clone()
    if periodic:
        both(E[0].movedim(1, 0)[:, :-1, 1:-1])
    both(E[1][:, :-1, 1:-1])
    both(E[2][:, 1:-1, :-1])
    both(E[0].movedim(2, 0)[:, :-1, :])
    both(E[1].movedim(2, 0)[:, :, :-1])
    if periodic:
        both(E[2].movedim(1, 0)[:, :, :-1])
    return E


def _interp(E, H, cell, f, shape):
    up = (f >= 0.5).to(f.dtype)
    low = {True: (torch.zeros_like(cell), 1.0 - f), False: (up.long(), 0.5 + up - f)}
    out = []
    for q in range(6):
        node = [(d == q) if q < 3 else (d != q - 3) for d in range(3)]
        at = [cell[:, d] + low[node[d]][0][:, d] for d in range(3)]
        w = [low[node[d]][1][:, d] for d in range(3)]
        A = (E[q] if q < 3 else H[q - 3]).reshape(-1)
        v = 0.0
        for b in range(8):
            o = (b >> 2, (b >> 1) & 1, b & 1)
            idx = ((at[0] + o[0]) * shape[1] + at[1] + o[1]) * shape[2] + at[2] + o[2]
            v = v + A[idx] * ((1 - w[0]) if o[0] else w[0]) * ((1 - w[1]) if o[1] else w[1]) * ((1 - w[2]) if o[2] else w[2])
        out.append(v)
    return torch.stack(out[:3], 1), torch.stack(out[3:], 1)


def _deposit(J, cell, xs, xe, iv, wt, shape):
    """one zigzag segment in cell units; iv 0 or 1 per axis: the cell-centre cell it lies in"""
    d = 0.5 * (xs + xe) - (iv.to(xs.dtype) - 0.5)
    D = xe - xs
    at = cell + iv
    low = 1.0 - d
    for comp in range(3):
        a, b = [q for q in range(3) if q != comp]
        s = D[:, a] * D[:, b] / 12.0
        for ha in (0, 1):
            for hb in (0, 1):
                o = [0, 0, 0]
                o[a], o[b] = ha, hb
                idx = ((at[:, 0] + o[0]) * shape[1] + at[:, 1] + o[1]) * shape[2] + at[:, 2] + o[2]
                w = (d[:, a] if ha else low[:, a]) * (d[:, b] if hb else low[:, b]) + (s if ha == hb else -s)
                J[comp] = J[comp].index_add(0, idx, wt[comp] * D[:, comp] * w)


def _push(case, part, E, H, J, shape, n, h, c):
    cell, f, p, m, q_m = part
    Ep, Hp = _interp(E, H, cell, f, shape)
    t = 0.5 * q_m * case["tau"]
    u = p + t * Ep
    b = t * Hp / torch.sqrt(1.0 + (u * u).sum(1, keepdim=True))
    s = u + torch.cross(u, b, dim=1)
    u = u + torch.cross(s, b, dim=1) * (2.0 / (1.0 + (b * b).sum(1, keepdim=True))) + t * Ep
    x1 = f + c * u / torch.sqrt(1.0 + (u * u).sum(1, keepdim=True))
    i1, i2 = (f >= 0.5).long(), (x1 >= 0.5).long()
    cross = i1 != i2
    D = x1 - f
    zero = torch.zeros_like(D)
    num, den = torch.where(cross, (0.5 - f) * D, zero).sum(1), torch.where(cross, D * D, zero).sum(1)
    hit = den > 0
    r = torch.where(hit, num / torch.where(hit, den, torch.ones_like(den)), torch.ones_like(num))
    x2 = torch.where(cross, torch.full_like(D, 0.5), f + D * r[:, None])
    wt = [m * h[d] / case["tau"] for d in range(3)]
    _deposit(J, cell, f, x2, i1, wt, shape)
    k = torch.nonzero(cross.any(1)).reshape(-1)
    if k.numel():
        _deposit(J, cell[k], x2[k], x1[k], i2[k], wt, shape)
    step = torch.floor(x1.detach())
    return [(cell + step.long()) % n, x1 - step, u, m, q_m]


def _advance(case, parts, E, H, dev, chunk=1 << 21):
    shape = (case["nx"] + 2, case["ny"] + 2, case["nz"] + 2)
    n = torch.tensor([case["nx"], case["ny"], case["nz"]], device=dev)
    h = (case["hx"], case["hy"], case["hz"])
    cf = [case["tau"] / v for v in h]
    c = torch.tensor(cf, dtype=torch.float64, device=dev)
    Q = _half_b(E, H, cf)
    H = [a + q for a, q in zip(H, Q)]
    J = [torch.zeros(shape[0] * shape[1] * shape[2], dtype=torch.float64, device=dev) for _ in range(3)]
    for s, part in enumerate(parts):
        size = part[0].shape[0]
        if size <= chunk:
            parts[s] = _push(case, part, E, H, J, shape, n, h, c)
            continue
        for a in range(0, size, chunk):
            z = _push(case, [v[a:a + chunk] for v in part[:3]] + part[3:], E, H, J, shape, n, h, c)
            for q in range(3):
                part[q][a:a + chunk] = z[q]
    J = _fold([a.reshape(shape) for a in J])
    H = [a + q for a, q in zip(H, Q)]
    E = _ghosts(_next_e(E, H, J, cf, case["tau"]), case["ghosts"] == "periodic")
    return E, H, J


def _rho(case, parts, dev):
    n = (case["nx"], case["ny"], case["nz"])
    shape = tuple(v + 2 for v in n)
    r = torch.zeros(shape[0] * shape[1] * shape[2], dtype=torch.float64, device=dev)
    for cell, f, _, m, _ in parts:
        up = (f >= 0.5).long()
        at, w = cell + up, f + 0.5 - up
        for b in range(8):
            o = (b >> 2, (b >> 1) & 1, b & 1)
            idx = ((at[:, 0] + o[0]) * shape[1] + at[:, 1] + o[1]) * shape[2] + at[:, 2] + o[2]
            v = 1.0
            for d in range(3):
                v = v * (w[:, d] if o[d] else 1.0 - w[:, d])
            r.index_add_(0, idx, m * v)
    r = r.reshape(shape)
    for d in range(3):
        v = r.movedim(d, 0)
        v[-2] = v[-2] + v[0]
        v[1] = v[1] + v[-1]
        v[0] = v[-2].clone()
        v[-1] = v[1].clone()
    return r


def _energy(parts, E, H):
    I = (slice(1, -1),) * 3
    e, b = (0.5 * sum(float((a[I] ** 2).sum()) for a in F) for F in (E, H))
    k = 0.0
    for _, _, p, m, q_m in parts:
        p2 = (p * p).sum(1)
        k += float((p2 / (torch.sqrt(1.0 + p2) + 1.0)).sum()) * (m / q_m)  # gamma - 1 without cancellation
    return [e, b, k, e + b + k]


def exact(case, seed):
    n = 3 * case["nx"] * case["ny"] * case["nz"] * case["ppc"]
    if case["stress"] or n * case["steps"] > (8.0e5 if case["kind"] == "grad" else 5.0e7):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    shape = (case["nx"] + 2, case["ny"] + 2, case["nz"] + 2)
    parts = _particles(case, int(seed), dev)
    E = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(3)]
    H = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(3)]
    I = (slice(1, -1),) * 3

    def flat(a):
        return a.detach().cpu().numpy().ravel()

    if case["kind"] == "audit":
        h = (case["hx"], case["hy"], case["hz"])
        r = _rho(case, parts, dev)
        E = [torch.from_numpy(a).reshape(shape).to(dev) for a in _smooth_fields(case, int(seed)).values()]
        div = sum((a - torch.roll(a, 1, d)) / h[d] for d, a in enumerate(E))
        G, G0 = torch.zeros_like(r), torch.zeros_like(r)
        G[I], G0[I] = (div - r)[I], -r[I]
        d = (G - G0)[I]
        check = [float(d.abs().max()), float(r[I].abs().max()), float((d * d).mean().sqrt()), float(G0.abs().max())]
        mom = [[float(v) for v in (p * (m / q_m)).sum(0)] for _, _, p, m, q_m in parts]
        return dict(fields=dict(rho=flat(r), residual=flat(G)), check=np.array(check), momentum=np.array(mom),
                    energy=np.array(_energy(parts, E, H)), energy_reference=sum(float((a * a).sum()) for a in E))
    if case["kind"] == "grad":
        beam = _species(case)[BEAM]
        p0 = parts[BEAM][2].clone().requires_grad_(True)
        parts[BEAM][2] = p0
        vol, hist = case["hx"] * case["hy"] * case["hz"], []
        for _ in range(case["steps"]):
            E, H, _J = _advance(case, parts, E, H, dev, chunk=1 << 40)
            hist.append(torch.stack([vol * (a[I] * a[I]).sum() for a in E]))
        L = sum(w[0] for w in hist[-_loss(case, beam)["window"]:])
        g, = torch.autograd.grad(L, p0)
        xi = p0.detach() - torch.tensor(beam["drift"], dtype=torch.float64, device=dev)
        order = torch.from_numpy(_bin_order(case)).to(dev)
        return dict(loss=np.array([float(L.detach())]), d_drift=flat(g.sum(0)), d_vth=np.array([float((g * xi).sum()) / beam["vth"]]),
                    d_p0=g[order].detach().cpu().numpy(), history=torch.stack(hist).detach().cpu().numpy())
    energies, history = [], []
    for _ in range(case["steps"]):
        E, H, J = _advance(case, parts, E, H, dev)
        if case["energies"]:
            energies.append(_energy(parts, E, H))
        history.append(sum(float((a * a).sum()) for a in E))
    out = dict(fields=dict(zip(EHJ, (flat(a) for a in E + H + J)), rho=flat(_rho(case, parts, dev))))
    if case["kind"] == "compute":
        out["history"] = np.array(history)
    elif case["energies"]:
        out["energies"] = np.array(energies)
    return out


def _bin_order(case):
    """The order of pic_get_particles after the generator: tiles of 8 x 4 x 8 cells (FP64 form) or 6 x 4 x 8 (FP32
    form), capped by the grid, each cell's particles together."""
    n = (case["nx"], case["ny"], case["nz"])
    t = (min(8 if case["precision"] == "fp64" else 6, n[0]), min(4, n[1]), 8 if n[2] >= 8 else (n[2] + 3) // 4 * 4)
    i, l, k = np.meshgrid(*[np.arange(v) for v in n], indexing="ij")
    i, l, k = i.ravel(), l.ravel(), k.ravel()
    cells = np.lexsort((k % t[2], l % t[1], i % t[0], k // t[2], l // t[1], i // t[0]))
    return (cells[:, None] * case["ppc"] + np.arange(case["ppc"])[None, :]).ravel()
