"""The work that a user of the particle-mesh framework has it do, as measurable cases.

Every case is a plain dict with a ``kind``:

* ``force``  -- one PM force evaluation (``gravity``), the layer every step of every run is made of;
* ``vjp``    -- the force and its adjoint (``gravity_vjp``), the layer of every reverse sweep;
* ``nbody``  -- a kick-drift-kick run (``nbody``), a user's plain simulation;
* ``model``  -- the differentiable run (``ForwardModel``): noise, 2LPT, steps, P(k) loss, gradients;
* ``lpt``    -- 2LPT initial conditions from linear modes;
* ``pk``     -- the P(k) loss of a particle set with its gradient;
* ``cic``    -- the deposit and the interpolation with per-particle values, and the adjoint of the latter;
* ``ensemble`` -- many small runs of uneven sizes advanced together.

Geometry: ``grid`` particles a side (``gy``, ``gz`` where they differ), a mesh ``factor`` times as fine,
2 Mpc/h between particles (the benchmark's resolution).  ``state`` says how far the particles have
moved: "early" is a smooth field of 0.4 spacings rms (a = 0.1), "late" one of 3 spacings rms with a
third of the Lagrangian patches fallen together (a = 1), "uniform" independent random positions.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pmpp_b200 as pb
from pmpp_b200 import lpt as pb_lpt
from pmpp_b200.ensemble import Ensemble
from pmpp_b200.pipeline import ForwardModel

SPACING = 2.0
OMEGA_M = 0.3
DEVICE = "cuda"


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest run of the repository's parity configuration: latency and launches count
        {"name": "force_64", "kind": "force", "grid": 64, "factor": 2.0, "state": "early", "dtype": "float32"},
        # the same particles in the float64 build, which users run for parity with their reference
        {"name": "force_64_f64", "kind": "force", "grid": 64, "factor": 2.0, "state": "late", "dtype": "float64"},
        # a usual size whose mesh (192) is no power of two, as in the ensembles
        {"name": "force_96", "kind": "force", "grid": 96, "factor": 2.0, "state": "late", "dtype": "float32"},
        # an ordinary production step, clustered as at a = 1
        {"name": "force_256", "kind": "force", "grid": 256, "factor": 2.0, "state": "late", "dtype": "float32"},
        # the benchmark's size
        {"name": "force_512", "kind": "force", "grid": 512, "factor": 2.0, "state": "late", "dtype": "float32"},
        # forward and adjoint of one force at an ordinary size
        {"name": "vjp_256", "kind": "vjp", "grid": 256, "factor": 2.0, "state": "late", "dtype": "float32"},
        # a whole small simulation: ten steps of the parity configuration
        {"name": "nbody_64", "kind": "nbody", "grid": 64, "factor": 2.0, "steps": 10, "dtype": "float32"},
        # the differentiable run end to end, gradients to the white noise and two parameters
        {"name": "model_128", "kind": "model", "grid": 128, "factor": 2.0, "steps": 4, "dtype": "float32"},
        # initial conditions at an ordinary size
        {"name": "lpt_256", "kind": "lpt", "grid": 256, "factor": 2.0, "dtype": "float32"},
        # the P(k) loss and its gradient at an ordinary size
        {"name": "pk_256", "kind": "pk", "grid": 256, "factor": 2.0, "state": "late", "dtype": "float32"},
        # a box of uneven sides and an odd mesh, three values per particle: deposits of momenta, forces
        # taken from a user's own meshes
        {"name": "cic_ragged", "kind": "cic", "grid": 100, "gy": 120, "gz": 90, "factor": 1.5, "channels": 3,
         "state": "late", "dtype": "float32"},
        # 24 members of three sizes, four steps, as a parameter sweep runs them
        {"name": "ensemble_24", "kind": "ensemble", "members": 24, "small": 32, "factor": 2.0, "steps": 4,
         "dtype": "float32"},
    ]


_USUAL = (32, 48, 64, 96, 128, 160, 192, 256)


def _side(rng, lo, hi):
    """A grid side in [lo, hi], over its logarithm: a usual size or any other, odd ones among them."""
    if rng.random() < 0.5:
        return rng.choice([s for s in _USUAL if lo <= s <= hi])
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["force", "force", "force", "vjp", "vjp", "nbody", "lpt", "pk", "cic", "cic"])
    case = {"kind": kind, "dtype": "float32"}
    if kind in ("force", "vjp"):
        case["grid"] = _side(rng, 32, 320 if kind == "force" else 256)
        case["factor"] = rng.choice([1.0, 2.0, 2.0, 2.0])
        case["state"] = rng.choice(["early", "late", "late", "uniform"])
        if kind == "force" and case["grid"] <= 128 and rng.random() < 0.2:
            case["dtype"] = "float64"
    elif kind == "nbody":
        case.update(grid=_side(rng, 32, 128), factor=rng.choice([1.0, 2.0]), steps=rng.randint(2, 10))
    elif kind == "lpt":
        case.update(grid=_side(rng, 32, 256), factor=rng.choice([1.0, 2.0]))
    elif kind == "pk":
        case.update(grid=_side(rng, 32, 256), factor=rng.choice([1.0, 2.0]), state=rng.choice(["early", "late"]))
    else:
        # sides in whole multiples of the mesh factor's denominator, so that the mesh has whole sides
        side = lambda: 2 * rng.randint(16, 96)
        case.update(grid=side(), gy=side(), gz=side(), factor=rng.choice([1.0, 1.5, 2.0]),
                    channels=rng.choice([1, 2, 3, 4]), state=rng.choice(["early", "late", "uniform"]))
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _shape(case):
    g = case["grid"]
    return (g, case.get("gy", g), case.get("gz", g))


def _mesh(case):
    return tuple(round(s * case["factor"]) for s in _shape(case))


def _schedule(case):
    """Scale factors of the run's steps, logarithmic as in the benchmark."""
    return np.geomspace(0.1, 1.0, case.get("steps", 1) + 1)


def _conf(case):
    return pb.Configuration(SPACING, _shape(case), _mesh(case), a_start=0.1, a_custom=_schedule(case),
                            float_dtype=case["dtype"], device=DEVICE)


def _gen(seed, k=0):
    return torch.Generator(device=DEVICE).manual_seed(1000003 * int(seed) + k)


def _smooth_modes(shape, seed, rms):
    """rFFT of a smooth random displacement field (three components), `rms` per component in units of
    the spacing: the spectrum of a density falling as k^-1.5 with k, cut at the smallest scales."""
    g = _gen(seed)
    f = torch.fft.rfftn(torch.randn((3, ) + shape, generator=g, device=DEVICE), dim=(1, 2, 3))
    k2 = sum(torch.meshgrid(*[(fr(n, device=DEVICE) * 2 * math.pi)**2 for fr, n in
                              zip((torch.fft.fftfreq, torch.fft.fftfreq, torch.fft.rfftfreq), shape)],
                            indexing="ij"))
    low = (2 * math.pi / 64)**2
    f = f * torch.where(k2 > 0, (k2 + low)**-0.9 * torch.exp(-k2 / 4), torch.zeros_like(k2))
    x = torch.fft.irfftn(f, s=shape, dim=(1, 2, 3))
    return x * (rms / x.std())


def _lattice(shape, mesh, dtype):
    """Anchors (int16) and displacements of the regular lattice, in mesh cells."""
    pm, dp = [], []
    for sp, sm in zip(shape, mesh):
        q = torch.arange(sp, device=DEVICE, dtype=torch.float64) * sm / sp
        pm.append(torch.round(q))
        dp.append(q - torch.round(q))
    pmid = torch.stack(torch.meshgrid(*pm, indexing="ij"), -1).reshape(-1, 3)
    off = torch.stack(torch.meshgrid(*dp, indexing="ij"), -1).reshape(-1, 3)
    return pmid.to(torch.int16).contiguous(), off.to(dtype)


def _particles(case, seed):
    """(pmid, disp) of the case's state."""
    shape, mesh = _shape(case), _mesh(case)
    dtype = torch.float64 if case["dtype"] == "float64" else torch.float32
    cell = SPACING * shape[0] / mesh[0]
    pmid, off = _lattice(shape, mesh, dtype)
    state = case.get("state", "early")
    n = pmid.shape[0]
    if state == "uniform":
        box = torch.tensor([s * SPACING for s in shape], device=DEVICE)
        move = torch.rand((n, 3), generator=_gen(seed, 1), device=DEVICE) * box - pmid * cell
        return pmid, move.to(dtype).contiguous()
    d = _smooth_modes(shape, seed, 0.4 if state == "early" else 3.0)
    if state == "late":
        # a third of the patches of 8^3 to 16^3 particles fall to a seventh of their size about their centres
        p = 8 if max(shape) < 96 else 16
        nb = [-(-s // p) for s in shape]
        hit = torch.rand(nb, generator=_gen(seed, 2), device=DEVICE) < 1 / 3
        ids = [torch.arange(s, device=DEVICE) for s in shape]
        m = hit[ids[0] // p][:, ids[1] // p][:, :, ids[2] // p]
        for a in range(3):
            c = (ids[a] % p - (p - 1) / 2.0).reshape([-1 if i == a else 1 for i in range(3)])
            centre = (ids[a] // p) * p + p // 2
            centre = torch.clamp(centre, max=shape[a] - 1)
            at = d[a].index_select(a, centre)
            d[a] = torch.where(m, at - (6.0 / 7.0) * c + (d[a] - at) / 7.0, d[a])
    disp = off * cell + (d.reshape(3, -1).T * SPACING).to(dtype)
    return pmid, disp.contiguous()


def _linear_modes(shape, seed):
    """Linear-density rFFT modes in the framework's units with a falling spectrum, rms density 1."""
    x = _smooth_modes(shape, seed, 1.0)[0]
    k2 = sum(torch.meshgrid(*[(fr(n, device=DEVICE) * 2 * math.pi)**2 for fr, n in
                              zip((torch.fft.fftfreq, torch.fft.fftfreq, torch.fft.rfftfreq), shape)],
                            indexing="ij"))
    delta = torch.fft.rfftn(x) * torch.sqrt(k2 + 1e-4)
    rms = torch.fft.irfftn(delta, s=shape).std()
    return (delta / rms * SPACING**3).to(torch.complex64).contiguous()


def _target(conf):
    """A fixed target spectrum: a power law in the shell number."""
    ns = math.floor(math.sqrt(3) * (conf.mesh_shape[0] // 2))
    return 2.0e4 * (1.0 + np.arange(ns) / 8.0)**-1.5


def _ensemble_specs(case, seed):
    rng = np.random.default_rng(int(seed))
    s = case["small"]
    sizes = (s, s * 3 // 2, 2 * s)
    n = case["members"]
    return [(sizes[k * 3 // n], float(rng.uniform(0.25, 0.35)), int(rng.integers(1, 2**31))) for k in range(n)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        confs, coss, ptcls = [], [], []
        for side, om, sd in _ensemble_specs(case, seed):
            sub = {"grid": side, "factor": case["factor"], "steps": case["steps"], "dtype": case["dtype"]}
            conf = _conf(sub)
            pmid, disp = _particles(sub, sd)
            confs.append(conf)
            coss.append(pb.boltzmann(pb.SimpleLCDM(conf, Omega_m=om)))
            ptcls.append(pb.Particles(conf, pmid, disp, (0.17 * (disp - disp.mean(0))).contiguous()))
        return {"kind": kind, "ens": Ensemble(confs, coss), "ptcls": ptcls}
    conf = _conf(case)
    s = {"kind": kind, "conf": conf}
    if kind in ("nbody", "model", "lpt"):
        s["cosmo"] = pb.boltzmann(pb.SimpleLCDM(conf, Omega_m=OMEGA_M))
    else:
        s["cosmo"] = pb.SimpleLCDM(conf, Omega_m=OMEGA_M)
    if kind == "lpt":
        s["modes"] = _linear_modes(_shape(case), seed)
        return s
    if kind == "model":
        g = _gen(seed)
        x = torch.randn(_shape(case), generator=g, device=DEVICE)
        s["omega"] = (torch.fft.rfftn(x) / math.sqrt(x.numel())).to(torch.complex64).contiguous()
        s["model"] = ForwardModel(conf, s["cosmo"])
        s["target"] = _target(conf)
        return s
    pmid, disp = _particles(case, seed)
    s["ptcl"] = pb.Particles(conf, pmid, disp)
    if kind == "nbody":
        s["ptcl"] = pb.Particles(conf, pmid, disp, (0.17 * (disp - disp.mean(0))).contiguous())
    elif kind == "vjp":
        s["cot"] = torch.randn(disp.shape, generator=_gen(seed, 3), device=DEVICE, dtype=disp.dtype)
    elif kind == "pk":
        s["target"] = _target(conf)
    elif kind == "cic":
        C = case["channels"]
        s["val"] = torch.randn((len(pmid), C), generator=_gen(seed, 3), device=DEVICE)
        s["mesh"] = torch.randn(_mesh(case) + (C, ), generator=_gen(seed, 4), device=DEVICE)
        s["cot"] = torch.randn((len(pmid), C), generator=_gen(seed, 5), device=DEVICE)
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "force":
        return pb.gravity(1.0, s["ptcl"], s["cosmo"], s["conf"])
    if kind == "vjp":
        dc, om = pb.gravity_vjp(1.0, s["ptcl"], s["cosmo"], s["conf"], s["cot"])
        return {"disp_cot": dc, "omega_m_cot": om}
    if kind == "nbody":
        out = pb.nbody(s["ptcl"], s["cosmo"], s["conf"])
        return {"disp": out.disp, "vel": out.vel, "acc": out.acc}
    if kind == "model":
        m = s["model"]
        final = m.forward(s["omega"])
        loss, g = m.loss(s["target"])
        grads = m.backward(g)
        return {"disp": final.disp, "loss": loss, "modes": grads["modes"], "omega_m": grads["Omega_m"],
                "a_s": grads["A_s_1e9"]}
    if kind == "lpt":
        p = pb_lpt.lpt(s["modes"], s["cosmo"], s["conf"])
        return {"disp": p.disp, "vel": p.vel}
    if kind == "pk":
        loss, g = pb.power_spectrum.pk_loss(s["ptcl"], s["conf"], s["target"])
        return {"loss": loss, "disp_cot": g}
    if kind == "cic":
        rho = pb.scatter(s["ptcl"], s["conf"], val=s["val"])
        got = pb.gather(s["ptcl"], s["conf"], s["mesh"])
        dc, mc = pb.gather_vjp(s["ptcl"], s["conf"], s["mesh"], s["cot"])
        return {"density": rho, "values": got, "disp_cot": dc, "mesh_cot": mc}
    outs = s["ens"].forward(s["ptcls"])
    return {"disp": [p.disp for p in outs[::6]], "vel": [p.vel for p in outs[::6]]}


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _fft_flops(cells):
    return 2.5 * cells * math.log2(cells)


def _force_work(n, cells, b):
    """One force: particles in, accelerations out, one real mesh written and read through one forward
    and three inverse transforms and read once more (each transform counted as one pass in, one out)."""
    return {"bytes": n * (6 + 3 * b + 3 * b) + cells * b * (1 + 8 + 3), "flops": 4 * _fft_flops(cells) + n * 250 + cells * 20}


def _add(*ws, times=1):
    return {k: times * sum(w[k] for w in ws) for k in ("bytes", "flops")}


def work(case):
    if case["kind"] == "ensemble":
        total = {"bytes": 0.0, "flops": 0.0}
        for side, _, _ in _ensemble_specs(case, 0):
            n, cells = side**3, round(side * case["factor"])**3
            total = _add(total, _add(_force_work(n, cells, 4), {"bytes": 48 * n, "flops": 12 * n},
                                     times=case["steps"] + 1))
        return total
    n, cells = math.prod(_shape(case)), math.prod(_mesh(case))
    b = 8 if case["dtype"] == "float64" else 4
    force = _force_work(n, cells, b)
    adjoint = {"bytes": n * 9 * b + cells * b * (3 + 3 + 8 + 1), "flops": 4 * _fft_flops(cells) + n * 500 + cells * 20}
    move = {"bytes": n * 12 * b, "flops": 12 * n}
    lpt = {"bytes": n * b * (2 + 2 * 13 + 12), "flops": 13 * _fft_flops(n) + 60 * n}
    pk = {"bytes": n * (6 + 3 * b) + cells * b * 4, "flops": _fft_flops(cells) + 60 * n + 20 * cells}
    kind = case["kind"]
    if kind == "force":
        return force
    if kind == "vjp":
        return _add(force, adjoint)
    if kind == "nbody":
        return _add(_add(force, move, times=case["steps"]), force)
    if kind == "lpt":
        return lpt
    if kind == "pk":
        return _add(pk, pk, {"bytes": 3 * b * n, "flops": 150 * n})
    if kind == "model":
        steps = case["steps"]
        return _add(lpt, lpt, pk, pk, _add(force, move, times=2 * steps + 1), _add(adjoint, move, times=steps + 1))
    C = case["channels"]
    one = n * (6 + 3 * b + C * b) + cells * C * b
    return {"bytes": 3 * one + n * (3 + C) * b + cells * C * b, "flops": n * C * 8 * 10.0}


# --------------------------------------------------------------------------
# how close another correct implementation comes
# --------------------------------------------------------------------------
def tolerance(case):
    """About four times the difference between the framework's two spectral routes (its own transforms and
    the library's) and between either and exact(), measured over the listed cases."""
    if case["dtype"] == "float64":
        return {"rel": 1e-12}
    kind = case["kind"]
    if kind in ("force", "lpt", "cic"):
        return {"rel": 2e-6}
    if kind in ("nbody", "ensemble"):
        return {"rel": 4e-6}
    if kind in ("vjp", "pk"):
        return {"rel": 2e-5}
    # model: positions that differ by rounding put a few particles in 1e5 across a cell face, where the
    # gradient of the deposit jumps; 1e-3 to 5e-3 of the modes' gradient was seen between the two routes
    return {"rel": 2e-2}


# --------------------------------------------------------------------------
# the same results in 64 bits
# --------------------------------------------------------------------------
F64 = torch.float64


def _corners(pmid, disp, cell, mesh, case):
    """Raveled indices and weights of the eight corners.  The position in cells is the quotient at the
    case's own precision, as the framework defines it (so that a particle near a cell face takes the same
    corners and one on a face the same, two-sided gradient); all that follows is in 64 bits."""
    at = disp.detach().to(getattr(torch, case["dtype"]))
    q = (at / torch.tensor(cell, dtype=at.dtype, device=at.device)).to(F64)
    low = torch.floor(q)
    f = (q - low) + (disp - disp.detach()) / cell
    base = pmid.to(torch.int64) + low.to(torch.int64)
    m = torch.tensor(mesh, device=disp.device)
    out = []
    for b in range(8):
        bit = torch.tensor([b & 1, (b >> 1) & 1, (b >> 2) & 1], device=disp.device)
        i = torch.remainder(base + bit, m)
        w = (1 - (f - bit).abs()).prod(-1)
        out.append(((i[:, 0] * mesh[1] + i[:, 1]) * mesh[2] + i[:, 2], w))
    return out


def _deposit(corners, mesh, val=1.0):
    rho = torch.zeros(math.prod(mesh), dtype=F64, device=DEVICE)
    for i, w in corners:
        rho = rho.index_add(0, i, w * val)
    return rho.reshape(mesh)


def _wave(mesh, spacing):
    ks = [torch.fft.fftfreq(n, device=DEVICE, dtype=F64) * (2 * math.pi / spacing) for n in mesh[:2]]
    ks.append(torch.fft.rfftfreq(mesh[2], device=DEVICE, dtype=F64) * (2 * math.pi / spacing))
    return ks


def _axis(k, a):
    return k.reshape([-1 if i == a else 1 for i in range(3)])


def _derivative(k, spacing):
    """Wavenumbers of a derivative: the Nyquist mode has none."""
    return torch.where((k.abs() - math.pi / spacing).abs() < 1e-6 * math.pi / spacing, torch.zeros_like(k), k)


def _accelerations(pmid, disp, case):
    mesh, shape = _mesh(case), _shape(case)
    cell = SPACING * shape[0] / mesh[0]
    cs = _corners(pmid, disp, cell, mesh, case)
    cells = math.prod(mesh)
    src = (_deposit(cs, mesh, cells / math.prod(shape)) - 1) * (1.5 * OMEGA_M)
    ks = _wave(mesh, cell)
    k2 = sum(_axis(k, a)**2 for a, k in enumerate(ks))
    G = torch.where(k2 > 0, -1 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
    if mesh != shape:  # modes beyond the particle lattice's Nyquist frequency are left out
        for a, k in enumerate(ks):
            G = G * _axis((k.abs() <= math.pi / SPACING * (1 + 1e-6)).to(F64), a)
    pot = torch.fft.rfftn(src) * G
    acc = []
    for a, k in enumerate(ks):
        F = torch.fft.irfftn(-1j * _axis(_derivative(k, cell), a) * pot, s=mesh).reshape(-1)
        acc.append(sum(w * F[i] for i, w in cs))
    return torch.stack(acc, -1)


def _growth(nodes, om):
    """First- and second-order growth D_m / a^m and their first two derivatives by ln a at the nodes,
    shape (order, derivative, node), by fourth-order Runge-Kutta steps in ln a from deep in matter
    domination (flat universe with a cosmological constant)."""
    def rhs(lna, g):
        a3 = np.exp(-3 * lna)
        e2 = om * a3 + 1 - om
        dlnh = -1.5 * om * a3 / e2
        o = 1.5 * om * a3 / e2
        return np.array([g[1], -(3 + dlnh - o) * g[0] - (4 + dlnh) * g[1],
                         g[3], o * g[0]**2 - (8 + 2 * dlnh - o) * g[2] - (6 + dlnh) * g[3]])

    t = math.log(0.5 * np.cbrt(np.finfo(np.float64).eps))
    g = np.array([1.0, 0.0, 3.0 / 7.0, 0.0])
    out = np.zeros((2, 3, len(nodes)))
    for j, a in enumerate(nodes):
        end = math.log(a) if a > 0 else t
        n = max(1, int(math.ceil((end - t) * 200)))
        h = (end - t) / n
        for _ in range(n if end > t else 0):
            k1 = rhs(t, g)
            k2 = rhs(t + h / 2, g + h / 2 * k1)
            k3 = rhs(t + h / 2, g + h / 2 * k2)
            k4 = rhs(t + h, g + h * k3)
            g, t = g + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4), t + h
        d = rhs(t, g)
        for m, (x, xp, xpp) in enumerate(((g[0], g[1], d[1]), (g[2], g[3], d[3])), 1):
            out[m - 1, :, j] = x, m * x + xp, m * m * x + 2 * m * xp + xpp
    return out


def _time_factors(a_steps, om):
    """Functions growth(a, order, derivative), drift(a_vel, a0, a1) and kick(a_acc, a0, a1); growth is
    interpolated linearly between the run's scale factors, as the time integrator defines it."""
    nodes = np.concatenate([np.linspace(0, a_steps[0], 1 + math.ceil(a_steps[0] * 128)), a_steps[1:]])
    tab = _growth(nodes, om)
    D = lambda a, m=1, d=0: a**m * np.interp(a, nodes, tab[m - 1, d])
    e2 = lambda a: om * a**-3 + 1 - om
    dlnh = lambda a: -1.5 * om * a**-3 / e2(a)
    gd = lambda a: a * a * math.sqrt(e2(a)) * D(a, 1, 1)
    gk = lambda a: a**3 * e2(a) * (D(a, 1, 2) + (2 + dlnh(a)) * D(a, 1, 1))
    return (D, lambda av, a0, a1: (D(a1) - D(a0)) / gd(av), lambda aa, a0, a1: (gd(a1) - gd(a0)) / gk(aa))


def _exact_nbody(case, seed):
    pmid, d32 = _particles(case, seed)
    disp = d32.to(F64)
    vel = (0.17 * (d32 - d32.mean(0))).to(F64)
    a = _schedule(case)
    _, drift, kick = _time_factors(a, OMEGA_M)
    acc = _accelerations(pmid, disp, case)
    for a0, a1 in zip(a[:-1], a[1:]):
        am = a0 * 0.5 + a1 * 0.5
        vel = vel + acc * kick(a0, a0, am)
        disp = disp + vel * drift(am, a0, a1)
        acc = _accelerations(pmid, disp, case)
        vel = vel + acc * kick(a1, am, a1)
    return {"disp": disp, "vel": vel, "acc": acc}


def _exact_lpt(case, seed):
    shape = _shape(case)
    pmid, off = _lattice(shape, _mesh(case), F64)
    cell = SPACING * shape[0] / _mesh(case)[0]
    modes = _linear_modes(shape, seed).to(torch.complex128) / SPACING**3
    ks = _wave(shape, SPACING)
    kd = [_derivative(k, SPACING) for k in ks]
    k2 = sum(_axis(k, a)**2 for a, k in enumerate(ks))
    G = torch.where(k2 > 0, -1 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
    p1 = modes * G
    strain = lambda i, j: torch.fft.irfftn(
        -(_axis(ks[i], i)**2 if i == j else _axis(kd[i], i) * _axis(kd[j], j)) * p1, s=shape)
    d = [strain(i, i) for i in range(3)]
    L = d[0] * d[1] + d[0] * d[2] + d[1] * d[2] - strain(0, 1)**2 - strain(0, 2)**2 - strain(1, 2)**2
    p2 = torch.fft.rfftn(L) * G
    D, _, _ = _time_factors(_schedule(case), OMEGA_M)
    a = 0.1
    h = a * a * math.sqrt(OMEGA_M * a**-3 + 1 - OMEGA_M)
    disp, vel = off * cell, torch.zeros_like(off)
    for m, p in ((1, p1), (2, p2)):
        g = torch.stack([torch.fft.irfftn(-1j * _axis(kd[i], i) * p, s=shape).reshape(-1) for i in range(3)], -1)
        disp = disp + D(a, m) * g
        vel = vel + h * D(a, m, 1) * g
    return {"disp": disp, "vel": vel}


def _exact_pk(case, seed):
    pmid, disp = _particles(case, seed)
    disp = disp.to(F64).requires_grad_(True)
    mesh, shape = _mesh(case), _shape(case)
    cell = SPACING * shape[0] / mesh[0]
    rho = _deposit(_corners(pmid, disp, cell, mesh, case), mesh)
    spec = torch.fft.rfftn(rho / rho.mean() - 1)
    n = [torch.fft.fftfreq(mesh[0], device=DEVICE, dtype=F64) * mesh[0],
         torch.fft.fftfreq(mesh[1], device=DEVICE, dtype=F64) * mesh[1],
         torch.arange(mesh[2] // 2 + 1, device=DEVICE, dtype=F64)]
    shells = math.floor(math.sqrt(3) * (mesh[0] // 2)) + 1
    r2 = sum(_axis(x, a)**2 for a, x in enumerate(n))
    shell = torch.clamp(torch.floor(torch.sqrt(r2) + 1e-9).to(torch.int64), max=shells - 1)
    mult = torch.full((mesh[2] // 2 + 1, ), 2.0, dtype=F64, device=DEVICE)
    mult[0] = 1
    if mesh[2] % 2 == 0:
        mult[-1] = 1
    w = math.prod(torch.sinc(_axis(x, a) / mesh[a]) for a, x in enumerate(n))
    p = (spec.real**2 + spec.imag**2) * w**-4 * mult
    sums = torch.zeros(shells, dtype=F64, device=DEVICE).index_add(0, shell.reshape(-1), p.reshape(-1))[1:]
    count = torch.bincount(torch.floor(torch.sqrt(r2) + 1e-6).to(torch.int64).reshape(-1),
                           weights=mult.expand(r2.shape).reshape(-1))[1:shells]
    pk = sums / count * (cell**3 / math.prod(mesh))
    t = torch.from_numpy(2.0e4 * (1.0 + np.arange(shells - 1) / 8.0)**-1.5).to(DEVICE)
    loss = (torch.log(pk / t)**2).mean()
    g, = torch.autograd.grad(loss, disp)
    return {"loss": loss.detach(), "disp_cot": g}


def _exact_cic(case, seed):
    pmid, disp = _particles(case, seed)
    mesh, shape, C = _mesh(case), _shape(case), case["channels"]
    n = len(pmid)
    val = torch.randn((n, C), generator=_gen(seed, 3), device=DEVICE).to(F64)
    field = torch.randn(mesh + (C, ), generator=_gen(seed, 4), device=DEVICE).to(F64).requires_grad_(True)
    cot = torch.randn((n, C), generator=_gen(seed, 5), device=DEVICE).to(F64)
    disp = disp.to(F64).requires_grad_(True)
    cs = _corners(pmid, disp, SPACING * shape[0] / mesh[0], mesh, case)
    rho = torch.stack([_deposit(cs, mesh, val[:, c]) for c in range(C)], -1).detach()
    flat = field.reshape(-1, C)
    got = sum(w[:, None] * flat[i] for i, w in cs)
    dc, mc = torch.autograd.grad((got * cot).sum(), (disp, field))
    return {"density": rho, "values": got.detach(), "disp_cot": dc, "mesh_cot": mc}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("model", "ensemble") or math.prod(_mesh(case)) > 700**3:
        return None
    with torch.set_grad_enabled(kind in ("vjp", "pk", "cic")):
        if kind == "force":
            pmid, disp = _particles(case, seed)
            return _accelerations(pmid, disp.to(F64), case)
        if kind == "vjp":
            pmid, disp = _particles(case, seed)
            cot = torch.randn(disp.shape, generator=_gen(seed, 3), device=DEVICE, dtype=disp.dtype).to(F64)
            disp = disp.to(F64).requires_grad_(True)
            dot = (_accelerations(pmid, disp, case) * cot).sum()
            g, = torch.autograd.grad(dot, disp)
            return {"disp_cot": g, "omega_m_cot": dot.detach() / OMEGA_M}
        if kind == "nbody":
            return _exact_nbody(case, seed)
        if kind == "lpt":
            return _exact_lpt(case, seed)
        if kind == "pk":
            return _exact_pk(case, seed)
        return _exact_cic(case, seed)
