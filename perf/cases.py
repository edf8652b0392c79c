"""What a user of this framework has it do, as measurable cases.

Six kinds of work, each through the public entry points that a program calls:

* ``flow``    -- a resident ``Engine`` advances one or more lattices by some steps; the program
  reads their statistics and state.  Arrested Newton flow, or RK4 dynamics (``dynamics``) with the
  FP64 energy audit.
* ``serve``   -- a request is admitted to an engine that already holds others, all advance by one
  serving chunk, the request's state is read and the request retired.
* ``view``    -- an interactive program's tick on a resident instance: one step, its statistics and
  the buffers that a renderer reads.
* ``step``    -- one ``Simulation.step``: the reference's own call on FP64 reference-layout buffers.
* ``observe`` -- energy, baryon number, centre of mass, radius (nuclear model: inertia tensors and
  shape too) and both density fields of a configuration.
* ``frame``   -- one frame of the headless viewer: the RGBA volume and its ray-march.

Theories, couplings, spacings, time steps and sizes are those of this repository's benchmark
configurations: a pion-only solve at 64^3, an omega solve at 128^3, Coulomb dynamics at 192^3, a
batch of pion and rho lattices, a serving stream of sides 48 to 192, with odd and ragged lattices
besides.  Fields are products of unit hedgehogs at random places with random isospin orientations,
with seeded noise for the pion-only model, inside a vacuum shell.

The state of an FP32 instance is returned in FP32 and that of an FP64 instance in FP64, the types
their flows are computed in.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from skyrmion_solver_b200 import theories
from skyrmion_solver_b200.core.simulation import Simulation
from skyrmion_solver_b200.engine import Engine

COMPONENTS = {"nuclear": 4, "omega": 5, "coulomb": 5, "rho": 13}
COUPLINGS = {
    "nuclear": {},
    "omega": dict(f_pi=139.8, m_pi=43.91, m_omega=249.5, beta_omega=8.036),
    "coulomb": dict(f_pi=105.9, m_pi=138.0, g=4.010, e=0.302822),
    "rho": dict(mpi=0.586, mrho=3.29, c_alpha=0.2256),
}
# multiplications and additions of one site's gradient (stencils and point arithmetic), roughly
GRADIENT_FLOPS = {"nuclear": 520, "omega": 300, "coulomb": 760, "rho": 2600}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an interactive program on a small FP32 lattice: latency and launches
        dict(name="view nuclear fp32 32", kind="view", theory="nuclear", precision="fp32", X=32, Y=32, Z=32, h=0.2),
        # the pion-only solve, in the serving default precision
        dict(name="flow nuclear fp64 64", kind="flow", theory="nuclear", precision="fp64", X=64, Y=64, Z=64, h=0.2,
             lumps=1, steps=16, dynamics=False, count=1),
        # the benchmark's solve: omega B = 4 at 128^3, compensated and defect-corrected FP32
        dict(name="flow omega fp32d 128", kind="flow", theory="omega", precision="fp32d", X=128, Y=128, Z=128,
             h=0.15, lumps=4, steps=16, dynamics=False, count=1),
        # a rho request of the serving stream in FP64, on a ragged lattice
        dict(name="flow rho fp64 ragged", kind="flow", theory="rho", precision="fp64", X=57, Y=50, Z=45, h=0.05,
             lumps=1, steps=8, dynamics=False, count=1),
        # boosted solitons, RK4 dynamics with the energy audit
        dict(name="dynamics coulomb fp32c 192", kind="flow", theory="coulomb", precision="fp32c", X=192, Y=192,
             Z=192, h=0.15, lumps=4, steps=10, dynamics=True, count=1),
        # batched relaxation of pion and rho lattices of uneven sizes
        dict(name="batch pion+rho fp32d", kind="flow", theory="nuclear+rho", precision="fp32d", X=64, Y=64, Z=64,
             h=0.2, lumps=2, steps=8, dynamics=False, count=6),
        # continuous batching: a request joins three others for one serving chunk
        dict(name="serve nuclear fp64 64", kind="serve", theory="nuclear", precision="fp64", X=64, Y=64, Z=64,
             h=0.2, lumps=1, steps=64, count=3),
        # the reference's own call: the pion-only configuration, the omega benchmark, a ragged lattice
        dict(name="step nuclear 64", kind="step", theory="nuclear", X=64, Y=64, Z=64, h=0.2, lumps=1),
        dict(name="step omega 128", kind="step", theory="omega", X=128, Y=128, Z=128, h=0.15, lumps=4),
        dict(name="step coulomb ragged", kind="step", theory="coulomb", X=75, Y=83, Z=61, h=0.15, lumps=2),
        # all observables of a relaxed configuration
        dict(name="observe nuclear 128", kind="observe", theory="nuclear", X=128, Y=128, Z=128, h=0.15, lumps=4),
        # a viewer frame at the viewer's default window size
        dict(name="frame nuclear 128", kind="frame", theory="nuclear", X=128, Y=128, Z=128, h=0.15, lumps=4,
             width=1200, height=900, display=2),
    ]


def _side(rng, lo, hi):
    """A lattice side: spread over the logarithm, half of them multiples of 16, else any size."""
    s = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(s / 16)) * 16 if rng.random() < 0.5 else int(round(s))))


def _sides(rng, lo, hi):
    if rng.random() < 0.5:
        s = _side(rng, lo, hi)
        return dict(X=s, Y=s, Z=s)
    return dict(X=_side(rng, lo, hi), Y=_side(rng, lo, hi), Z=_side(rng, lo, hi))


def draw(rng):
    kind = rng.choices(["flow", "dynamics", "batch", "serve", "view", "step", "observe", "frame"],
                       [30, 8, 8, 8, 8, 22, 10, 6])[0]
    theory = rng.choices(["nuclear", "omega", "coulomb", "rho"], [40, 30, 15, 15])[0]
    h = 0.05 if theory == "rho" else rng.choice([0.1, 0.15, 0.2])
    top = 72 if theory == "rho" else 160
    precision = rng.choices(["fp64", "fp32d", "fp32c", "fp32"], [40, 35, 10, 15])[0]
    if kind == "flow":
        sides = _sides(rng, 32, top)
        steps = rng.choice([8, 16, 20]) if sides["X"] * sides["Y"] * sides["Z"] < 2_000_000 else 8
        return dict(kind="flow", theory=theory, precision=precision, **sides, h=h,
                    lumps=1 if theory == "rho" else rng.randint(1, 4), steps=steps, dynamics=False, count=1)
    if kind == "dynamics":
        theory = "nuclear" if theory == "rho" else theory
        return dict(kind="flow", theory=theory, precision=rng.choice(["fp32c", "fp64"]), **_sides(rng, 48, 144),
                    h=0.15, lumps=rng.randint(2, 4), steps=10, dynamics=True, count=1)
    if kind == "batch":
        s = _side(rng, 48, 72)
        precision = rng.choice(["fp64", "fp32d"])
        return dict(kind="flow", theory="nuclear+rho", precision=precision, X=s, Y=s, Z=s, h=0.2,
                    lumps=rng.randint(1, 3), steps=8, dynamics=False,
                    count=rng.randint(3, 6 if precision == "fp32d" else 4))
    if kind == "serve":
        s = 48 if theory == "rho" else _side(rng, 48, 64)
        return dict(kind="serve", theory=theory, precision=rng.choice(["fp64", "fp32d"]), X=s, Y=s, Z=s, h=h, lumps=1,
                    steps={"nuclear": 64, "rho": 16}.get(theory, 32), count=1 if theory == "rho" else rng.randint(1, 3))
    if kind == "view":
        return dict(kind="view", theory=theory, precision=precision, **_sides(rng, 24, 64), h=h)
    sides = _sides(rng, 32, top)
    lumps = 1 if theory == "rho" else rng.randint(1, 4)
    if kind == "frame":
        s = _side(rng, 48, 128)
        return dict(kind="frame", theory="nuclear", X=s, Y=s, Z=s, h=0.15, lumps=lumps,
                    width=rng.randint(400, 1200), height=rng.randint(300, 900), display=rng.choice([1, 2]))
    return dict(kind=kind, theory=theory, **sides, h=h, lumps=lumps)


# ---------------------------------------------------------------------------
# inputs, in plain torch
# ---------------------------------------------------------------------------
def _members(case):
    """The lattices of a case: (theory, sides) in the order of admission.  The lattices of a batch
    take the base size and larger ones in steps of 8, pion and rho in turn."""
    names = case["theory"].split("+")
    s = (case["X"], case["Y"], case["Z"])
    n = case.get("count", 1)
    if case["kind"] == "serve":  # the residents, then the request
        return [(names[0], tuple(v + 8 * (k % 2) for v in s)) for k in range(n)] + [(names[0], s)]
    return [(names[k % len(names)], tuple(v + 8 * (k // len(names)) for v in s)) for k in range(n)]


def _params(case, theory, dims):
    h = case["h"]
    factor = 0.1 if case.get("dynamics") else (0.05 if theory == "rho" else 0.2)
    th = theories.by_short_name(theory)
    prm = th.params.default_params(
        xlen=dims[0], ylen=dims[1], zlen=dims[2], lsx=h, lsy=h, lsz=h, xsize=h * (dims[0] - 1),
        ysize=h * (dims[1] - 1), zsize=h * (dims[2] - 1), time_step=factor * h,
        killkinen=not case.get("dynamics", False), **COUPLINGS[theory])
    return th, prm


class _Constants:
    """Couplings and lattice constants, as plain numbers."""

    def __init__(self, case, theory, dims):
        self.h = float(case["h"])
        self.vol = self.h ** 3
        self.dt = (0.1 if case.get("dynamics") else (0.05 if theory == "rho" else 0.2)) * self.h
        self.kill = not case.get("dynamics", False)
        c = COUPLINGS[theory]
        if theory == "nuclear":
            self.c = (1.0, 1.0)
        elif theory == "omega":
            self.c = (c["m_pi"] / c["m_omega"], c["m_omega"] * c["beta_omega"] / c["f_pi"])
        elif theory == "coulomb":
            self.c = (2.0 * c["m_pi"] / (c["g"] * c["f_pi"]), c["g"] ** 2 * c["e"] ** 2 / 2.0)
        else:
            self.c = (c["mpi"], c["mrho"], c["c_alpha"])


def _quaternion_product(a, b):
    return torch.stack([a[0] * b[0] - a[1] * b[1] - a[2] * b[2] - a[3] * b[3],
                        a[0] * b[1] + a[1] * b[0] + a[2] * b[3] - a[3] * b[2],
                        a[0] * b[2] - a[1] * b[3] + a[2] * b[0] + a[3] * b[1],
                        a[0] * b[3] + a[1] * b[2] - a[2] * b[1] + a[3] * b[0]])


def _field(case, theory, dims, seed):
    """FP64 field (C, X, Y, Z) and velocity (zero, or the boost of a dynamics case)."""
    rnd = random.Random(seed)
    h = case["h"]
    gen = torch.Generator(device="cuda").manual_seed(rnd.getrandbits(40))
    ax = [(torch.arange(n, dtype=torch.float64, device="cuda") - (n - 1) / 2.0) * h for n in dims]
    x, y, z = torch.meshgrid(*ax, indexing="ij")
    half = [h * (n - 1) / 2.0 for n in dims]
    scale = min(1.5, 0.3 * min(half))
    places = []
    while len(places) < case.get("lumps", 1):
        c = [rnd.uniform(-0.4, 0.4) * v if case.get("lumps", 1) > 1 else rnd.uniform(-0.05, 0.05) * v for v in half]
        far = 0.4 * min(half) * 0.98 ** rnd.randint(0, 60)
        if all(math.dist(c, p) > far for p in places) or rnd.random() < 0.02:
            places.append(c)
    phi = None
    for c in places:
        q = [rnd.gauss(0.0, 1.0) for _ in range(4)]
        nq = math.sqrt(sum(v * v for v in q))
        w, i, j, k = (v / nq for v in q)
        rot = [[1 - 2 * (j * j + k * k), 2 * (i * j - w * k), 2 * (i * k + w * j)],
               [2 * (i * j + w * k), 1 - 2 * (i * i + k * k), 2 * (j * k - w * i)],
               [2 * (i * k - w * j), 2 * (j * k + w * i), 1 - 2 * (i * i + j * j)]]
        d = (x - c[0], y - c[1], z - c[2])
        r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2).clamp_min(1e-12)
        f = math.pi * torch.exp(-r / scale)
        s = torch.sin(f) / r
        lump = torch.stack([torch.cos(f)] + [s * (m[0] * d[0] + m[1] * d[1] + m[2] * d[2]) for m in rot])
        phi = lump if phi is None else _quaternion_product(phi, lump)
    if theory == "nuclear":  # the pion-only configuration's noise
        phi = phi + 1e-3 * (2.0 * torch.rand(phi.shape, dtype=torch.float64, device="cuda", generator=gen) - 1.0)
    phi /= torch.sqrt((phi * phi).sum(0))
    field = torch.zeros((COMPONENTS[theory],) + tuple(dims), dtype=torch.float64, device="cuda")
    field[:4] = phi
    shell = torch.ones(dims, dtype=torch.bool, device="cuda")
    shell[2:-2, 2:-2, 2:-2] = False
    field[:, shell] = 0.0
    field[0, shell] = 1.0
    if theory == "omega":  # the omega field starts as -c_omega times the baryon density
        k = _Constants(case, theory, dims)
        field[4] = -k.c[1] * _baryon(field, k) / k.vol
    velocity = torch.zeros_like(field)
    if case.get("dynamics"):
        slope = _first(field[:4], 0, h)
        v = -(0.15 * torch.tanh(-x)) * slope
        v -= (v * field[:4]).sum(0) * field[:4]
        v[:, shell] = 0.0
        velocity[:4] = v
    return field, velocity


def _reads(precision):
    """The type in which an instance's state is returned."""
    return torch.float64 if precision == "fp64" else torch.float32


def prepare(case, seed):
    kind = case["kind"]
    members = _members(case) if kind in ("flow", "serve") else [(case["theory"], (case["X"], case["Y"], case["Z"]))]
    s = {"kind": kind, "case": case}
    built = []
    for k, (theory, dims) in enumerate(members):
        th, prm = _params(case, theory, dims)
        built.append((theory, dims, th, prm) + _field(case, theory, dims, 1000 * seed + k))
    if kind in ("flow", "serve", "view"):
        s["engine"] = Engine(0)
        s["ids"], s["out"] = [], []
        residents = built[:-1] if kind == "serve" else built
        for theory, dims, th, prm, field, velocity in residents:
            s["ids"].append(s["engine"].add(th, prm, field, velocity if case.get("dynamics") else None,
                                            precision=case["precision"]))
        for _, _, _, _, field, _ in (built[-1:] if kind == "serve" else built):
            s["out"].append((torch.empty_like(field), torch.empty_like(field)))
        if kind == "serve":
            s["request"] = built[-1][2:5]
        return s
    theory, dims, th, prm, field, _ = built[0]
    if kind == "frame":
        k = _Constants(case, theory, dims)
        r = th.render_headless.Renderer(case["width"], case["height"], dims[2])
        r.bind_params(*th.params.pack_device_params(prm.resolved()), device=0)
        r.set_display_mode(case["display"])
        s.update(renderer=r, field=field.reshape(-1).contiguous(), density=_baryon(field, k).reshape(-1).contiguous())
        return s
    sim = Simulation(prm, th)
    sim.initialize({"mode": "vacuum"})
    sim.Field.copy_(field.reshape(-1))
    s["sim"] = sim
    s["energy"] = float(sim.observables()["energy"]) if kind == "step" else None
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _numbers(st, to):
    return torch.tensor([st.energy, st.baryon, st.gabs], dtype=to)


def run(s):
    return {"flow": _run_flow, "serve": _run_serve, "view": _run_view, "step": _run_step, "observe": _run_observe,
            "frame": _run_frame}[s["kind"]](s)


def _run_flow(s):
    case, eng = s["case"], s["engine"]
    to = _reads(case["precision"])
    eng.step(case["steps"])
    stats = eng.stats_all()
    got = []
    for i, (f, v) in zip(s["ids"], s["out"]):
        eng.read_device(i, f, v)
        got.append({"field": f.to(to), "velocity": v.to(to), "stats": _numbers(stats[i], to)})
        if case["dynamics"]:
            got[-1]["hamiltonian"] = torch.tensor(eng.audit(i)["hamiltonian"], dtype=to)
    return got


def _run_serve(s):
    case, eng = s["case"], s["engine"]
    to = _reads(case["precision"])
    th, prm, field = s["request"]
    i = eng.add(th, prm, field, None, precision=case["precision"])
    eng.step(case["steps"])
    stats = eng.stats_all()
    f, v = s["out"][0]
    eng.read_device(i, f, v)
    eng.remove(i)
    return {"field": f.to(to), "velocity": v.to(to), "stats": _numbers(stats[i], to),
            "residents": [_numbers(stats[j], to) for j in s["ids"]]}


def _run_view(s):
    case, eng = s["case"], s["engine"]
    to = _reads(case["precision"])
    eng.step(1)
    st = eng.stats(s["ids"][0])
    field, density = eng.view(s["ids"][0])
    return {"field": field.to(to), "density": density.to(to), "stats": _numbers(st, to)}


def _run_step(s):
    sim = s["sim"]
    s["energy"], err = sim.step(s["energy"])
    return {"field": sim.Field, "velocity": sim.Velocity, "gradient": sim.EnergyGradient, "energy": s["energy"],
            "err": err}


def _run_observe(s):
    sim = s["sim"]
    out = dict(sim.observables())
    out["center"] = sim.compute_center_of_mass()
    out["radius"] = sim.compute_rms_radius()
    if s["case"]["theory"] == "nuclear":
        out["U"] = sim.compute_U_tensor()
        out["V"] = sim.compute_V_tensor()
        out["W"] = sim.compute_W_tensor()
        out["Q"] = sim.compute_quadrupole_tensor()
        out["D"] = sim.compute_D_term()
    sim.compute_energy_density()
    g, b = sim._launch()
    sim.kernels.compute_skyrmion_number_kernel[g, b](sim.entmp, sim.Field, None, sim.p_i_d, sim.p_f_d)
    out["energy_density"], out["baryon_density"] = sim.en, sim.entmp
    return out


def _run_frame(s):
    r = s["renderer"]
    image = r.render(density_flat=s["density"], field_flat=s["field"])
    return {"volume": r.volume, "image": image}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("flow", "serve", "view"):
        members = _members(case) if kind != "view" else [(case["theory"], (case["X"], case["Y"], case["Z"]))]
        size = 8 if case["precision"] == "fp64" else 4
        low = 1 if case["precision"] in ("fp32c", "fp32d") else 0
        steps = case.get("steps", 1)
        b = f = 0.0
        for theory, dims in members:
            n, c = float(np.prod(dims)), COMPONENTS[theory]
            b += steps * (4 + 2 * low) * c * size * n  # field and velocity in and out of every step
            f += steps * 4 * GRADIENT_FLOPS[theory] * n
        n, c = float(np.prod(members[-1][1])), COMPONENTS[members[-1][0]]
        return {"bytes": b + 2 * 8 * c * n, "flops": f}
    n, c = float(case["X"]) * case["Y"] * case["Z"], COMPONENTS[case["theory"]]
    if kind == "step":  # reads F and V; writes F, V, the stage slopes k1..k4 and l1..l4, the stage input, the gradient
        return {"bytes": 14 * 8 * c * n, "flops": 4 * GRADIENT_FLOPS[case["theory"]] * n}
    if kind == "observe":  # reads the field, writes two densities
        return {"bytes": 8 * (c + 2) * n, "flops": (12 * c + 150 + (700 if case["theory"] == "nuclear" else 0)) * n}
    # frame: density and pion field in, RGBA volume out; about 500 lit samples of 60 operations per pixel
    return {"bytes": 48 * n + 16.0 * case["width"] * case["height"], "flops": 3.0e4 * case["width"] * case["height"]}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _shift(f, axis, k):
    """f moved so that index i holds f[i + k] along a lattice axis; zeros come in."""
    ax = f.dim() - 3 + axis
    out = torch.zeros_like(f)
    n = f.shape[ax]
    if abs(k) < n:
        out.narrow(ax, max(0, -k), n - abs(k)).copy_(f.narrow(ax, max(0, k), n - abs(k)))
    return out


def _inside(f, axis, low):
    """1 inside the lattice by `low` sites below and 2 above along an axis, else 0."""
    n = f.shape[f.dim() - 3 + axis]
    m = torch.zeros(n, dtype=f.dtype, device=f.device)
    m[low:n - 2] = 1.0
    return m.reshape([n if a == axis else 1 for a in range(3)])


def _first(f, axis, h):
    d = (8.0 * (_shift(f, axis, 1) - _shift(f, axis, -1)) - (_shift(f, axis, 2) - _shift(f, axis, -2))) / (12.0 * h)
    return d * _inside(f, axis, 2)


def _second(f, axis, h):
    d = (16.0 * (_shift(f, axis, 1) + _shift(f, axis, -1)) - (_shift(f, axis, 2) + _shift(f, axis, -2)) -
         30.0 * f) / (12.0 * h * h)
    return d * _inside(f, axis, 2)


def _mixed(f, a, b, h):
    def raw(g, axis):
        return _shift(g, axis, -2) - _shift(g, axis, 2) + 8.0 * (_shift(g, axis, 1) - _shift(g, axis, -1))
    return raw(raw(f, a), b) / (144.0 * h * h) * _inside(f, a, 3) * _inside(f, b, 3)


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2] + a[3] * b[3]


def _cross4(a, u, v):
    def p(i, j):
        return u[i] * v[j] - u[j] * v[i]
    return torch.stack([a[1] * p(2, 3) - a[2] * p(1, 3) + a[3] * p(1, 2),
                        -(a[0] * p(2, 3) - a[2] * p(0, 3) + a[3] * p(0, 2)),
                        a[0] * p(1, 3) - a[1] * p(0, 3) + a[3] * p(0, 1),
                        -(a[0] * p(1, 2) - a[1] * p(0, 2) + a[2] * p(0, 1))])


def _minus_det(phi, D):
    return _dot(_cross4(phi, D[1], D[2]), D[0])


def _baryon(F, k):
    D = [_first(F[:4], i, k.h) for i in range(3)]
    return _minus_det(F[:4], D) * k.vol / (2.0 * math.pi ** 2)


def _sidx(i, j):
    return i if i == j else 2 + i + j


def _eps(i, j, k):
    return 0 if len({i, j, k}) < 3 else (1 if (i, j, k) in ((0, 1, 2), (1, 2, 0), (2, 0, 1)) else -1)


def _quartic(D, S):
    """sum over i != j of the Skyrme term's variation, for the four pion components."""
    n = [_dot(d, d) for d in D]
    acc = sum((n[0] + n[1] + n[2] - n[i]) * S[i][:4] for i in range(3))
    for i, j in ((0, 1), (0, 2), (1, 2)):
        s = S[_sidx(i, j)]
        acc = acc + (_dot(D[j], s) - _dot(S[j], D[i])) * D[i][:4] + (_dot(D[i], s) - _dot(S[i], D[j])) * D[j][:4] \
            - 2.0 * _dot(D[i], D[j]) * s[:4]
    return acc


def _coupling(phi, D):
    out = 0.0
    for i, j, m in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        out = out + 2.0 * D[i][4] * _cross4(phi, D[j], D[m])
    return out


def _gradient(theory, F, k):
    D = [_first(F, i, k.h) for i in range(3)]
    S = [_second(F, i, k.h) for i in range(3)]
    if theory != "omega":
        S += [_mixed(F, 0, 1, k.h), _mixed(F, 0, 2, k.h), _mixed(F, 1, 2, k.h)]
    phi = F[:4]
    lap = S[0] + S[1] + S[2]
    g = torch.empty_like(F)
    if theory == "nuclear":
        g[:4] = -lap - k.c[1] ** 2 * _quartic(D, S)
        g[0] -= k.c[0] ** 2
    elif theory == "omega":
        g[:4] = -0.25 * lap[:4] + k.c[1] / (4.0 * math.pi ** 2) * _coupling(phi, D)
        g[0] -= 0.25 * k.c[0] ** 2
        g[4] = F[4] - lap[4] + k.c[1] * _minus_det(phi, D) / (2.0 * math.pi ** 2)
    elif theory == "coulomb":
        g[:4] = -lap[:4] - _quartic(D, S)
        g[0] -= k.c[0] ** 2
        g[:4] -= k.c[1] / (4.0 * math.pi ** 2) * _coupling(phi, D)
        g[4] = -k.c[1] * (lap[4] + _minus_det(phi, D) / (2.0 * math.pi ** 2))
    else:
        _gradient_rho(F, D, S, k, g)
    g[:4] -= _dot(g, phi) * phi
    return g


def _r(i, a):
    return 4 + 3 * i + a


def _gradient_rho(F, D, S, k, g):
    mpi, mrho, ca = k.c
    g[:4] = -2.0 * (S[0] + S[1] + S[2])[:4] - 2.0 * _quartic(D, S)
    g[0] -= 2.0 * mpi ** 2

    def dR(a, j, m, l):
        return S[_sidx(j, l)][_r(m, a)] - S[_sidx(m, l)][_r(j, a)]
    for a in range(3):
        for j in range(3):
            r = sum(dR(a, i, j, i) for i in range(3) if i != j)
            g[0] += 16.0 * ca * D[j][a + 1] * r
            g[a + 1] -= 16.0 * ca * D[j][0] * r
            for b in range(3):
                for c in range(3):
                    if _eps(a, b, c):
                        g[b + 1] += 16.0 * ca * _eps(a, b, c) * D[j][c + 1] * r
    for a in range(3):
        for i in range(3):
            val = 8.0 * mrho ** 2 * F[_r(i, a)]
            for j in range(3):
                if j == i:
                    continue
                sij, sjj = S[_sidx(i, j)], S[j]
                om = sij[0] * D[j][a + 1] + D[i][0] * sjj[a + 1] - sij[a + 1] * D[j][0] - D[i][a + 1] * sjj[0]
                for b in range(3):
                    for c in range(3):
                        if _eps(a, b, c):
                            om = om + _eps(a, b, c) * (sij[b + 1] * D[j][c + 1] + D[i][b + 1] * sjj[c + 1])
                val = val + 8.0 * dR(a, i, j, j) - 16.0 * ca * om
            g[_r(i, a)] = val


def _energy(theory, F, k):
    D = [_first(F, i, k.h) for i in range(3)]
    n = [_dot(d, d) for d in D]
    two = n[0] + n[1] + n[2]
    four = sum(n[i] * n[j] - _dot(D[i], D[j]) ** 2 for i, j in ((0, 1), (0, 2), (1, 2)))
    if theory == "nuclear":
        e = 0.5 * two + 0.5 * k.c[1] ** 2 * four + k.c[0] ** 2 * (1.0 - F[0])
    elif theory == "omega":
        e = 0.125 * two + 0.25 * k.c[0] ** 2 * (1.0 - F[0]) + 0.5 * F[4] ** 2 + 0.5 * sum(d[4] ** 2 for d in D)
    elif theory == "coulomb":
        e = two + four + 2.0 * k.c[0] ** 2 * (1.0 - F[0]) + 0.5 * k.c[1] * sum(d[4] ** 2 for d in D)
    else:
        mpi, mrho, ca = k.c
        e = two + four + 2.0 * mpi ** 2 * (1.0 - F[0]) + 4.0 * mrho ** 2 * (F[4:] ** 2).sum(0)
        for a in range(3):
            for i in range(3):
                for j in range(3):
                    if i == j:
                        continue
                    R = D[i][_r(j, a)] - D[j][_r(i, a)]
                    om = D[i][0] * D[j][a + 1] - D[i][a + 1] * D[j][0]
                    for b in range(3):
                        for c in range(3):
                            if _eps(a, b, c):
                                om = om + _eps(a, b, c) * D[i][b + 1] * D[j][c + 1]
                    e = e + 2.0 * R * R - 8.0 * ca * R * om
    return e * k.vol


def _hamiltonian(theory, F, V, k):
    """The energy that the RK4 dynamics conserves: for omega and Coulomb the auxiliary field enters
    with the opposite sign and its coupling to the baryon density."""
    e, sign = _energy(theory, F, k), [1.0] * F.shape[0]
    if theory in ("omega", "coulomb"):
        D4 = sum(_first(F[4], i, k.h) ** 2 for i in range(3))
        sign[4] = -1.0
        if theory == "omega":
            aux = k.vol * 0.5 * (F[4] ** 2 + D4)
            e = e - 2.0 * aux - k.c[1] * F[4] * _baryon(F, k)
        else:
            aux = k.vol * 0.5 * k.c[1] * D4
            e = 0.5 * (e - aux) - aux + k.c[1] * F[4] * _baryon(F, k)
    return float(e.sum()) + 0.5 * k.vol * sum(s * float((v * v).sum()) for s, v in zip(sign, V))


def _rk4(theory, F, V, k):
    """One RK4 step: the new field and velocity, and the gradient at the last stage's input."""
    l1 = -k.dt * _gradient(theory, F, k)
    l2 = -k.dt * _gradient(theory, F + 0.5 * k.dt * V, k)
    l3 = -k.dt * _gradient(theory, F + 0.5 * k.dt * (V + 0.5 * l1), k)
    g = _gradient(theory, F + k.dt * (V + 0.5 * l2), k)
    Fn = F + k.dt * (V + (l1 + l2 + l3) / 6.0)
    Vn = V + (l1 + 2.0 * l2 + 2.0 * l3 - k.dt * g) / 6.0
    Fn[:4] /= torch.sqrt(_dot(Fn, Fn))
    Vn[:4] -= _dot(Vn, Fn) * Fn[:4]
    return Fn, Vn, g


def _flow(case, theory, dims, seed, steps):
    k = _Constants(case, theory, dims)
    F, V = _field(case, theory, dims, seed)
    E = float(_energy(theory, F, k).sum())
    g = None
    for _ in range(steps):
        F, V, g = _rk4(theory, F, V, k)
        new = float(_energy(theory, F, k).sum())
        if k.kill and new > E:
            V = torch.zeros_like(V)
        E = new
    out = {"field": F, "velocity": V, "stats": torch.tensor([E, float(_baryon(F, k).sum()), float(g.abs().max())],
                                                            dtype=torch.float64)}
    if case.get("dynamics"):
        out["hamiltonian"] = torch.tensor(_hamiltonian(theory, F, V, k), dtype=torch.float64)
    return out, g


def _shape(F, k, dims):
    """Centre of mass, radius and the nuclear model's inertia, quadrupole and D-term sums."""
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") * k.h for n in dims]
    grid = torch.stack(torch.meshgrid(*ax, indexing="ij"))
    b = _baryon(F, k)
    B = float(b.sum())
    com = np.array([float((b * x).sum()) for x in grid]) / B
    r = grid - torch.tensor(com, device="cuda").reshape(3, 1, 1, 1)
    r2 = (r * r).sum(0)
    out = {"center": com, "radius": math.sqrt(max(float((b.abs() * r2).sum()) / B, 0.0))}
    D = torch.stack([_first(F[:4], i, k.h) for i in range(3)])
    sg, pi = F[0], F[1:4]
    eps = torch.tensor([[[float(_eps(i, j, m)) for m in range(3)] for j in range(3)] for i in range(3)],
                       dtype=torch.float64, device="cuda")
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    L = sg * D[:, 1:] - pi * D[:, :1] + torch.einsum("abc,bxyz,kcxyz->kaxyz", eps, pi, D[:, 1:])
    T = pi[:, None] * pi[None] - eye[:, :, None, None, None] * (pi * pi).sum(0) + \
        sg * torch.einsum("iab,bxyz->iaxyz", eps, pi)
    LL = torch.einsum("iaxyz,jaxyz->ijxyz", L, L)
    TT = torch.einsum("iaxyz,jaxyz->ijxyz", T, T)
    LT = torch.einsum("iaxyz,jaxyz->ijxyz", T, L)
    k2, tr = k.c[1] ** 2, LL[0, 0] + LL[1, 1] + LL[2, 2]

    def mul(a, c):
        return torch.einsum("imxyz,mjxyz->ijxyz", a, c)
    A = LL + k2 * (LL * tr - mul(LL, LL))
    Bm = LT + k2 * (LT * tr - mul(LT, LL))
    U = TT + k2 * (TT * tr - torch.einsum("imxyz,jmxyz->ijxyz", LT, LT))
    rr = torch.einsum("ilm,lxyz->imxyz", eps, r)  # rr[i, m] v_m = (r x v)_i
    V = torch.einsum("imxyz,mpxyz,jpxyz->ijxyz", rr, A, rr)
    W = torch.einsum("jmxyz,imxyz->ijxyz", rr, Bm)
    out["U"], out["V"], out["W"] = (2.0 * k.vol * t.sum((2, 3, 4)).cpu().numpy() for t in (U, V, W))
    Q = (3.0 * r[:, None] * r[None] - eye[:, :, None, None, None] * r2) * (0.5 * b)
    out["Q"] = Q.sum((2, 3, 4)).cpu().numpy()
    four = sum(LL[i, i] * LL[j, j] - LL[i, j] ** 2 for i, j in ((0, 1), (0, 2), (1, 2)))
    e = 0.5 * tr + 0.5 * k2 * four + k.c[0] ** 2 * (1.0 - sg)
    S = LL + k2 * (tr * LL - mul(LL, LL)) - eye[:, :, None, None, None] * e
    trS = S[0, 0] + S[1, 1] + S[2, 2]
    stress = torch.einsum("ixyz,jxyz,ijxyz->xyz", r, r, S) - r2 * trS / 3.0
    out["D"] = -0.4 * float(_energy("nuclear", F, k).sum()) * float(stress.sum()) * k.vol
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("flow", "serve"):
        got = []
        for n, (theory, dims) in enumerate(_members(case)):
            got.append(_flow(case, theory, dims, 1000 * seed + n, case["steps"])[0])
        if kind == "flow":
            return got
        return dict(got[-1], residents=[g["stats"] for g in got[:-1]])
    theory, dims = case["theory"], (case["X"], case["Y"], case["Z"])
    k = _Constants(case, theory, dims)
    if kind == "view":
        out, _ = _flow(case, theory, dims, 1000 * seed, 1)
        return {"field": out["field"].reshape(-1), "density": _baryon(out["field"], k).reshape(-1),
                "stats": out["stats"]}
    if kind == "step":
        out, g = _flow(case, theory, dims, 1000 * seed, 1)
        return {"field": out["field"].reshape(-1), "velocity": out["velocity"].reshape(-1), "gradient": g.reshape(-1),
                "energy": float(out["stats"][0]), "err": float(g.max())}
    F, _ = _field(case, theory, dims, 1000 * seed)
    if kind == "observe":
        e, b = _energy(theory, F, k), _baryon(F, k)
        out = {"energy": float(e.sum()), "skyrmion_number": float(b.sum()), "energy_density": e.reshape(-1),
               "baryon_density": b.reshape(-1)}
        more = _shape(F, k, dims) if theory == "nuclear" else _center(b, k, dims)
        return dict(out, **more)
    d = _baryon(F, k)  # frame: the volume; the image's early exits have no value of their own in 64 bits
    norm = torch.sqrt((F[1:4] ** 2).sum(0))
    flat = norm * norm <= 1e-20
    n = F[1:4] / torch.where(flat, torch.ones_like(norm), norm)
    n[:, flat] = 0.0
    n[2][flat] = 1.0
    vol = torch.cat([((d - d.min()) / (d.max() - d.min() + 1e-30))[None], n])
    return {"volume": vol.permute(3, 2, 1, 0).contiguous(), "image": None}


def _center(b, k, dims):
    ax = [torch.arange(n, dtype=torch.float64, device="cuda") * k.h for n in dims]
    grid = torch.stack(torch.meshgrid(*ax, indexing="ij"))
    B = float(b.sum())
    com = np.array([float((b * x).sum()) for x in grid]) / B
    r2 = ((grid - torch.tensor(com, device="cuda").reshape(3, 1, 1, 1)) ** 2).sum(0)
    return {"center": com, "radius": math.sqrt(max(float((b.abs() * r2).sum()) / B, 0.0))}
