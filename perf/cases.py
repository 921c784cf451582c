"""What a user of the solver has it do, as timed cases: time-step runs over the range of grid sizes,
a whole job from host buffers, the batched launch, the adjoint gradient and the reference's whole
run behind marchingLoop's parameter list.

``listed()`` names the cases, ``draw`` makes more of the same ranges, ``prepare`` builds what a
program has in hand before the call, ``run`` is one pass through the public Python entry points,
``work`` the bytes and operations of a pass, and ``exact`` the same results from a plain 64-bit
update written here in torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from fdtd_gb300 import scenario as S
from fdtd_gb300 import solver

EX, EY, EZ, HX, HY, HZ = range(6)

# ------------------------------------------------------------------------------------------------
# Cases
# ------------------------------------------------------------------------------------------------


def _run_case(name, nx, ny, nz, steps, pml=(10,) * 6, boxes=0, sources=1, probes=1, resistors=0, magnetic=False,
              aniso=False):
    c = dict(kind="run", nx=nx, ny=ny, nz=nz, steps=steps, boxes=boxes, sources=sources, probes=probes,
             resistors=resistors, magnetic=magnetic, aniso=aniso)
    c.update({"p%d" % q: int(v) for q, v in enumerate(pml)})
    if name:
        c["name"] = name
    return c


def listed():
    cases = [
        # One step at a time with the fields looked at after each: an interactive or coupled program.
        _run_case("vacuum64_one_step", 64, 64, 64, 1),
        # The small workload (64^3 vacuum, one source, one probe): a run whose launches count.
        _run_case("vacuum64_run", 64, 64, 64, 200),
        # An odd small structure with a different CPML on every face (one face without), a lumped
        # load and per-axis and magnetic materials: what a reference user's own geometry looks like.
        _run_case("ragged_93x77x51", 93, 77, 51, 100, pml=(6, 10, 8, 0, 12, 5), boxes=8, sources=2, probes=6,
                  resistors=1, magnetic=True, aniso=True),
        # Random-box workloads, from a component-sized grid to the HBM-sized domain.
        _run_case("boxes128", 128, 128, 128, 50, boxes=32, sources=4, probes=16),
        _run_case("boxes_225x190x163", 225, 190, 163, 24, pml=(8, 8, 10, 10, 12, 12), boxes=32, sources=2, probes=16),
        _run_case("boxes256", 256, 256, 256, 24, boxes=64, sources=4, probes=16),
        _run_case("boxes512", 512, 512, 512, 20, boxes=64, sources=4, probes=16),
        _run_case("boxes_1024x1024x896", 1024, 1024, 896, 8, boxes=64, sources=4, probes=16),
    ]
    # The whole job of a batch system: handle, index and waveforms from host memory, steps, probes.
    job = _run_case("job_boxes256", 256, 256, 256, 32, boxes=64, sources=4, probes=16)
    job["kind"] = "job"
    cases.append(job)
    # A parameter sweep: independent instances of uneven sizes advanced together.
    cases.append(dict(name="batch64", kind="batch", n=64, lo=32, hi=96, layout=5, steps=32, pml=8, boxes=8))
    # One iteration of a gradient optimisation: start state, new permittivities, forward, backward.
    cases.append(dict(name="adjoint128", kind="adjoint", n=128, dx=32, dy=32, dz=16, pml=10, steps=192, every=64))
    # The reference's own program: marchingLoop on a microstrip patch, with plates and a port.
    cases.append(dict(name="microstrip", kind="marching", X=60, Y=100, Z=16, steps=400, pml=8, air=6, width=6,
                      current=2, resistor=0))
    return cases


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["job", "batch", "adjoint", "marching"])
    if kind in ("run", "job"):
        cells = _log_uniform(rng, 6.4e4, 4e8 if kind == "run" else 6e7)
        edge = cells ** (1 / 3)
        pml = [rng.choice([0, 4, 6, 8, 10, 10, 10, 12, 15]) for _ in range(6)]
        if rng.random() < 0.6:
            pml = [rng.choice([6, 8, 10, 10, 12])] * 6
        dims = [max(40, int(edge * rng.uniform(0.6, 1.5))) for _ in range(3)]
        if rng.random() < 0.3:
            dims[0] = dims[0] // 32 * 32
        n = dims[0] * dims[1] * dims[2]
        steps = max(1, min(rng.choice([1, 7, 20, 64, 200]), int(1.2e9 / n)))
        c = _run_case(None, dims[0], dims[1], dims[2], steps, pml, boxes=rng.choice([0, 8, 32, 64]),
                      sources=rng.choice([1, 2, 4]), probes=rng.choice([1, 6, 16]), resistors=rng.choice([0, 0, 1]),
                      magnetic=rng.random() < 0.25, aniso=rng.random() < 0.25)
        c["kind"] = kind
        return c
    if kind == "batch":
        lo = rng.choice([32, 40, 48])
        return dict(kind="batch", n=rng.choice([2, 8, 24, 48]), lo=lo, hi=lo + rng.choice([4, 20, 48]),
                    layout=rng.randrange(1000), steps=rng.choice([5, 16, 40]), pml=rng.choice([6, 8, 10]), boxes=8)
    if kind == "adjoint":
        n = rng.choice([48, 57, 72, 96, 120])
        return dict(kind="adjoint", n=n, dx=rng.randint(4, n // 4), dy=rng.randint(4, n // 4), dz=rng.randint(4, n // 5),
                    pml=rng.choice([6, 8, 10]), steps=rng.randint(60, 160), every=rng.choice([0, 16, 64]))
    return dict(kind="marching", X=rng.randint(40, 72), Y=rng.randint(60, 110), Z=rng.randint(8, 18),
                steps=rng.randint(60, 400), pml=rng.choice([6, 8, 10]), air=rng.choice([4, 6]), width=rng.choice([4, 6, 9]),
                current=rng.choice([2, 2, 3]), resistor=rng.choice([0, 1]))


# ------------------------------------------------------------------------------------------------
# Scenarios from a case and a seed
# ------------------------------------------------------------------------------------------------

WAVE = 4096  # samples of a source waveform (a pulse train, so that later steps are driven too)


def _pulses(dt, delay):
    one = S.gaussian_derivative(512, dt, 30e9, 1e-3, delay_steps=delay)
    return np.resize(one, WAVE).astype(np.float32)


def _scenario(case, seed):
    """The grid of a run case: dielectric boxes, sources, loads and probes at seeded places outside
    the CPML."""
    rng = np.random.default_rng([seed, 11])
    n = (case["nx"], case["ny"], case["nz"])
    pml = tuple(case["p%d" % q] for q in range(6))
    delta = (1e-3, 1e-3, 1e-3)
    dt = S.courant_dt(*delta, 0.99)
    lo = [max(1, pml[2 * a]) for a in range(3)]
    hi = [n[a] - max(1, pml[2 * a + 1]) - 1 for a in range(3)]
    mats, bricks = [S.Material()], []
    for b in range(case["boxes"]):
        start = [int(rng.integers(lo[a], max(lo[a] + 1, hi[a] - 1))) for a in range(3)]
        size = [int(rng.integers(max(2, (hi[a] - lo[a]) // 32), max(4, (hi[a] - lo[a]) // 4))) for a in range(3)]
        end = [min(start[a] + size[a], hi[a]) for a in range(3)]
        eps, sig, mu, sm = float(rng.uniform(1, 12)), float(rng.uniform(0, 0.05)), 1.0, float(S.REF_TINY)
        if case["magnetic"] and b % 3 == 1:
            mu, sm = float(rng.uniform(1, 3)), float(rng.uniform(1, 500))
        if case["aniso"] and b % 3 == 2:
            eps = tuple(float(v) for v in rng.uniform(1, 12, 3))
        mats.append(S.Material(eps_r=eps, sigma_e=sig, mu_r=mu, sigma_m=sm))
        bricks.append(S.Brick((*start, *end), len(mats) - 1))
    used, sources, loads, probes = set(), [], [], []

    def place(margin):
        while True:
            q = tuple(int(rng.integers(lo[a] + margin, max(lo[a] + margin + 1, hi[a] - margin))) for a in range(3))
            if q not in used:
                used.add(q)
                return q

    for _ in range(case["sources"]):
        i, j, k = place(2)
        sources.append(S.LumpedSource((i, j, k, i, j, k + 1), 50.0, _pulses(dt, float(rng.uniform(0, 40)))))
    for _ in range(case["resistors"]):
        i, j, k = place(2)
        loads.append(S.Resistor((i, j, k, i, j, k + 1), 50.0))
    for q in range(case["probes"]):
        i, j, k = place(2)
        probes.append(S.Probe(EZ if q % 2 == 0 else HX, i, j, k))
    return S.Scenario("case", *n, *delta, float(dt), pml, case["steps"], mats, bricks, sources, loads, probes)


def _start_fields(nx, ny, nz, seed, device):
    """A state in mid-run: noise of the size of a propagating wave in every cell, zero on the outer
    planes (the domain's walls). Six float32 fields, one at a time."""
    gen = torch.Generator(device=device)
    for c in range(6):
        gen.manual_seed(1000 * seed + c)
        f = torch.rand((nz, ny, nx), generator=gen, device=device, dtype=torch.float32)
        f.sub_(0.5).mul_(1.0 if c < 3 else 1.0 / 377.0)
        for d in range(3):
            f.select(d, 0).zero_()
            f.select(d, f.shape[d] - 1).zero_()
        yield c, f


def _batch_scenarios(case, seed):
    dims = np.random.default_rng([case["layout"], 3]).integers(case["lo"], case["hi"] + 1, size=(case["n"], 3))
    out = []
    for q, d in enumerate(dims):
        c = _run_case(None, int(d[0]), int(d[1]), int(d[2]), case["steps"], (case["pml"],) * 6, boxes=case["boxes"])
        out.append(_scenario(c, 7919 * seed + q))
    return out


def _design(case, seed):
    n, c = case["n"], case["n"] // 2
    d = (case["dx"], case["dy"], case["dz"])
    dt = S.courant_dt(1e-3, 1e-3, 1e-3, 0.99)
    src = S.LumpedSource((n // 4, c, c, n // 4, c, c + 1), 50.0, S.gaussian_derivative(case["steps"], dt, 30e9, 1e-3))
    sc = S.Scenario("design", n, n, n, 1e-3, 1e-3, 1e-3, float(dt), (case["pml"],) * 6, case["steps"], [S.Material()], [],
                    [src], [], [])
    box = tuple(c - d[a] // 2 for a in range(3)) + tuple(c - d[a] // 2 + d[a] for a in range(3))
    eps = np.random.default_rng([seed, 4]).uniform(1.0, 12.0, size=d[::-1]).astype(np.float32)
    return sc, box, eps, (3 * n // 4, c, c)


def _microstrip(case, seed):
    """marchingLoop's parameters of a patch on a grounded substrate with a feed strip."""
    f = np.float32
    rng = np.random.default_rng([seed, 9])
    X, Y, Z, P, A, W = (case[q] for q in ("X", "Y", "Z", "pml", "air", "width"))
    dx, dy, dz = f(0.389e-3), f(0.4e-3), f(0.265e-3)
    eps_0, mu_0, pi, c = S.REF_EPS0, S.REF_MU0, S.REF_PI, S.ref_light_speed()
    dt = S.courant_dt(dx, dy, dz, 0.99)
    tau = f(f(f(20) * dy) / (f(2) * c))
    s0, s1 = X // 2 - W // 2, X // 2 - W // 2 + W  # feed strip columns
    p0, p1, pj0, pj1 = X // 5, X - X // 5, Y // 2, Y - Y // 8  # patch
    eps_r = float(f(rng.uniform(2.0, 6.0)))
    a = dict(NUMDEV=1, eps_0=eps_0, pi=pi, mu_0=mu_0, c=c, dx=dx, dy=dy, dz=dz, dt=dt, X=X, Y=Y, Z=Z,
             n_t_steps=case["steps"], source_tp=1, source_freq=f(2e9), source_amp=f(rng.uniform(0.5, 2.0)),
             source_min_x=s0 * dx, source_min_y=f(0), source_min_z=f(0), source_max_x=s1 * dx, source_max_y=f(0),
             source_max_z=3 * dz, source_direction=3, rs=f(50), nc=f(20), tau=tau, t_0=f(f(3) * tau))
    for q in "xyz":
        for side in "np":
            a["pml_%s_%s" % (q, side)] = P
            a["air_buff_%s_%s" % (q, side)] = A
    a.update(brick_min_x=[0.0], brick_min_y=[0.0], brick_min_z=[0.0], brick_max_x=[X * dx], brick_max_y=[Y * dy],
             brick_max_z=[3 * dz], brick_opt=1, brick_num=1)
    for q in "xyz":
        a.update({"brick_sigma_e_" + q: [4e-4], "brick_eps_r_" + q: [eps_r], "brick_sigma_m_" + q: [1.2e-38],
                  "brick_mu_r_" + q: [1.0], "pec_sigma_e_" + q: [1e10] * 3})
    a.update(pec_min_x=[0.0, s0 * dx, p0 * dx], pec_min_y=[0.0, 0.0, pj0 * dy], pec_min_z=[0.0, 3 * dz, 3 * dz],
             pec_max_x=[X * dx, s1 * dx, p1 * dx], pec_max_y=[Y * dy, pj0 * dy, pj1 * dy], pec_max_z=[0.0, 3 * dz, 3 * dz],
             pec_opt=1, pec_num=3)
    a.update(resistor_min_x=p1 * dx, resistor_min_y=pj1 * dy, resistor_min_z=f(0), resistor_max_x=p1 * dx,
             resistor_max_y=pj1 * dy, resistor_max_z=3 * dz, resistor_resist=f(50), resistor_direction=3,
             resistor_opt=case["resistor"])
    vj = Y // 6
    zlo = 0 if case["current"] == 3 else 3
    a.update(sampled_voltage_min_x=s0 * dx, sampled_voltage_min_y=vj * dy, sampled_voltage_min_z=f(0),
             sampled_voltage_max_x=s1 * dx, sampled_voltage_max_y=vj * dy, sampled_voltage_max_z=3 * dz, voltage_direction=3,
             sampled_current_min_x=s0 * dx, sampled_current_min_y=vj * dy, sampled_current_min_z=zlo * dz,
             sampled_current_max_x=s1 * dx, sampled_current_max_y=vj * dy, sampled_current_max_z=3 * dz,
             current_direction=case["current"])
    return a


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------


def _fields_of(sim, out):
    for c in range(6):
        sim.get_field_device(c, out[c].data_ptr())
    return out


def _simulation(sc, seed):
    sim = solver.Simulation.from_scenario(sc)
    for c, f in _start_fields(sc.nx, sc.ny, sc.nz, seed, "cuda"):
        sim.set_field_device(c, f.data_ptr())
        torch.cuda.current_stream().synchronize()  # f is freed next
    sim.prepare()
    return sim


def prepare(case, seed):
    torch.cuda.init()
    kind = case["kind"]
    if kind == "run":
        sc = _scenario(case, seed)
        out = torch.empty((6, sc.nz, sc.ny, sc.nx), dtype=torch.float32, device="cuda")
        return dict(kind=kind, sim=_simulation(sc, seed), steps=case["steps"], out=out)
    if kind == "job":
        sc = _scenario(case, seed)
        index = torch.from_numpy(sc.material_index()).pin_memory()
        out = torch.empty((6, sc.nz, sc.ny, sc.nx), dtype=torch.float32, device="cuda")
        return dict(kind=kind, sc=sc, index=index, steps=case["steps"], out=out)
    if kind == "batch":
        scs = _batch_scenarios(case, seed)
        sims = [_simulation(sc, 7919 * seed + q) for q, sc in enumerate(scs)]
        sizes = [6 * sc.cells for sc in scs]
        flat = torch.empty(sum(sizes), dtype=torch.float32, device="cuda")
        outs = [v.view(6, sc.nz, sc.ny, sc.nx) for v, sc in zip(flat.split(sizes), scs)]
        return dict(kind=kind, sims=sims, batch=solver.Batch(sims), steps=case["steps"], flat=flat, outs=outs)
    if kind == "adjoint":
        sc, box, eps, probe = _design(case, seed)
        sim = solver.Simulation.from_scenario(sc)
        sim.set_design_region(box, eps)
        sim.prepare()
        start = torch.empty(sim.state_bytes(), dtype=torch.uint8, device="cuda")
        sim.save_state(start.data_ptr())
        return dict(kind=kind, sim=sim, box=box, eps=eps, probe=probe, steps=case["steps"], every=case["every"],
                    start=start)
    return dict(kind=kind, params=_microstrip(case, seed))


def run(state):
    kind = state["kind"]
    if kind == "run":
        sim, n = state["sim"], state["steps"]
        sim.step(n)
        _fields_of(sim, state["out"])
        return [sim.read_probes(sim.current_step - n, n), state["out"]]
    if kind == "job":
        n = state["steps"]
        with solver.Simulation.from_scenario(state["sc"], material_index=state["index"].numpy(), probe_capacity=n) as sim:
            sim.step(n)
            _fields_of(sim, state["out"])
            return [sim.read_probes(0, n), state["out"]]
    if kind == "batch":
        state["batch"].step(state["steps"])
        state["batch"].synchronize()
        for sim, out in zip(state["sims"], state["outs"]):
            _fields_of(sim, out)
        return state["flat"]
    if kind == "adjoint":
        sim = state["sim"]
        sim.load_state(state["start"].data_ptr())
        sim.set_design_region(state["box"], state["eps"])
        J = sim.adjoint_forward(state["steps"], state["probe"], state["every"])
        return [J, sim.adjoint_backward()]
    return list(solver.marching_loop(state["params"]))


# ------------------------------------------------------------------------------------------------
# Work of one pass
# ------------------------------------------------------------------------------------------------


def _step_work(n, pml):
    """(bytes, flops) of one time step: every field component read and written once and the material
    byte, and each CPML memory value read and written (two arrays for E and two for H per slab)."""
    cells = n[0] * n[1] * n[2]
    psi = 4 * sum((pml[2 * a] + pml[2 * a + 1]) * cells // n[a] for a in range(3))
    return 49 * cells + 8 * psi, 42 * cells + 5 * psi


def work(case):
    kind = case["kind"]
    if kind in ("run", "job"):
        n = (case["nx"], case["ny"], case["nz"])
        b, f = _step_work(n, [case["p%d" % q] for q in range(6)])
        cells = n[0] * n[1] * n[2]
        extra = 24 * cells + (cells if kind == "job" else 0)  # the fields handed out; the index uploaded
        return {"bytes": b * case["steps"] + extra, "flops": f * case["steps"]}
    if kind == "batch":
        tot = {"bytes": 0, "flops": 0}
        for sc in _batch_scenarios(case, 0):
            b, f = _step_work((sc.nx, sc.ny, sc.nz), sc.pml)
            tot["bytes"] += b * case["steps"] + 24 * sc.cells
            tot["flops"] += f * case["steps"]
        return tot
    if kind == "adjoint":
        # the forward, and the transposed update once per step (as many fields and CPML memory)
        b, f = _step_work((case["n"],) * 3, (case["pml"],) * 6)
        design = 24 * case["dx"] * case["dy"] * case["dz"]  # the design region's E kept and read per step
        return {"bytes": (2 * b + design) * case["steps"], "flops": 2 * f * case["steps"]}
    n = [case[q] + 2 * (case["pml"] + case["air"]) for q in "XYZ"]
    b, f = _step_work(n, (case["pml"],) * 6)
    return {"bytes": b * case["steps"], "flops": f * case["steps"]}


# ------------------------------------------------------------------------------------------------
# The same results in 64 bits
# ------------------------------------------------------------------------------------------------


def _profile(n, pn, pp, delta, dt, eps0, mu0, pi):
    """1-D CPML profiles {kappa, b, a} for E and H (cubic grading, kappa_max 5, alpha_max 0.05)."""
    out = {m: [np.ones(n), np.zeros(n), np.zeros(n)] for m in "eh"}
    s_max = 1.5 * 4.0 / (150.0 * pi * delta)
    for q in list(range(pn)) + list(range(n - pp, n)):
        for m, off in (("e", 0.75), ("h", 0.25)):
            ro = (pn - q - off) / pn if q < pn else (q - (n - pp - 1) - off) / pp
            scale, c0 = (1.0, eps0) if m == "e" else (mu0 / eps0, mu0)
            s, al, ka = s_max * ro ** 3 * scale, 0.05 * (1 - ro) * scale, 1 + 4 * ro ** 3
            b = math.exp(-(dt / c0) * (s / ka + al))
            out[m][0][q], out[m][1][q] = ka, b
            out[m][2][q] = (b - 1) * s / (ka * (s + ka * al)) / delta
    return out


class _Exact:
    """The Yee step with CPML in float64: state = six fields, then the twelve CPML memories."""

    def __init__(self, sc, device, design=None, edges=None):
        f8 = dict(dtype=torch.float64, device=device)
        n = (sc.nx, sc.ny, sc.nz)
        d = [float(np.float32(v)) for v in (sc.dx, sc.dy, sc.dz)]
        self.dt = dt = float(np.float32(sc.dt))
        eps0, mu0, pi = (float(np.float32(v)) for v in (sc.eps0, sc.mu0, sc.pi))
        self.d, self.shape, self.device = d, (sc.nz, sc.ny, sc.nx), device
        self.prof = {}
        for a in range(3):
            p = _profile(n[a], sc.pml[2 * a], sc.pml[2 * a + 1], d[a], dt, eps0, mu0, pi)
            view = [1, 1, 1]
            view[2 - a] = n[a]
            for m in "eh":
                ka, b, c = (torch.tensor(v, **f8).view(view) for v in p[m])
                self.prof[m, a] = (1.0 / (ka * d[a]), b, c)
        index = torch.zeros(self.shape, dtype=torch.uint8)
        for bk in sc.bricks:
            i0, j0, k0, i1, j1, k1 = bk.box
            index[k0:k1, j0:j1, i0:i1] = bk.material
        index = index.to(device).long()
        mats = torch.tensor(np.array([m.axes() for m in sc.materials]).astype(np.float64), **f8)  # (m, axis, property)
        self.ca, self.cb, self.inject = [], [], []

        def shift(t, dim):  # the cell one below along a dimension (its own value at the low wall)
            return torch.cat([t.narrow(dim, 0, 1), t.narrow(dim, 0, t.shape[dim] - 1)], dim)

        for c in range(3):
            eps, sig = mats[:, c, 0][index], mats[:, c, 1][index]
            if design is not None:
                (i0, j0, k0, i1, j1, k1), e = design
                pad = (i0, n[0] - i1, j0, n[1] - j1, k0, n[2] - k1)
                eps = eps * torch.nn.functional.pad(torch.zeros_like(e), pad, value=1.0) + torch.nn.functional.pad(e, pad)
            p, q = [2 - a for a in range(3) if a != c]
            eps = (eps + shift(eps, p)) / 2
            eps = (eps + shift(eps, q)) / 2
            sig = (sig + shift(sig, p)) / 2
            sig = (sig + shift(sig, q)) / 2
            for comp, i0, j0, i1, j1, k, s in edges or ():  # edges of zero-thickness plates
                if comp == c:
                    sig[k, j0:j1 + 1, i0:i1 + 1] = s
            den, num = 2 * eps * eps0 + dt * sig, 2 * eps * eps0 - dt * sig
            lumped = [(s, s.waveform) for s in sc.sources] + [(r, None) for r in sc.resistors] if c == 2 else []
            for s, wave in lumped:
                i0, j0, k0, i1, j1, k1 = s.box
                box = (slice(k0, k1), slice(j0, j1 + 1), slice(i0, i1 + 1))
                area = (1 + i1 - i0) * (1 + j1 - j0) / (k1 - k0) * float(np.float32(s.resistance)) * d[0] * d[1]
                add = torch.zeros_like(den)
                add[box] = dt * d[2] / area
                den, num = den + add, num - add
                if wave is not None:
                    self.inject.append((box, -2 * dt / area / den[box].detach(), np.asarray(wave, np.float64) / (k1 - k0)))
            mask = torch.zeros(self.shape, **f8)
            mask[tuple(slice(0 if a == c else 1, n[a] - 1) for a in (2, 1, 0))] = 1.0
            self.ca.append(1.0 + mask * (num / den - 1.0))
            self.cb.append(mask * (2 * dt) / den)
        for c in range(3):
            mu, sm = mats[:, c, 2][index], mats[:, c, 3][index]
            mu1, sm1 = shift(mu, 2 - c), shift(sm, 2 - c)
            mu, sm = 2 * mu * mu1 / (mu + mu1), 2 * sm * sm1 / (sm + sm1)
            mu.select(2 - c, 0).fill_(1.0)  # faces on the low wall keep the free-space values
            sm.select(2 - c, 0).fill_(0.0)
            den, num = 2 * mu * mu0 + dt * sm, 2 * mu * mu0 - dt * sm
            mask = torch.zeros(self.shape, **f8)
            mask[tuple(slice(0, n[a] if a == c else n[a] - 1) for a in (2, 1, 0))] = 1.0
            self.ca.append(1.0 + mask * (num / den - 1.0))
            self.cb.append(mask * (2 * dt) / den)

    def start(self, fields=None):
        z = lambda: torch.zeros(self.shape, dtype=torch.float64, device=self.device)  # noqa: E731
        return [z() if fields is None else fields[c] for c in range(6)] + [z() for _ in range(12)]

    def step(self, s, m):
        s, half = list(s), {}
        for base, other, kind in ((0, 3, "e"), (3, 0, "h")):
            new = []
            for c in range(3):
                # component c takes +d(other[c+2])/d(c+1) - d(other[c+1])/d(c+2) for E, the reverse for H
                u, v = (c + 1) % 3, (c + 2) % 3
                total = None
                for t, (axis, src, sign) in enumerate(((u, v, 1.0), (v, u, -1.0))):
                    f, dim = s[other + src], 2 - axis
                    edge = torch.zeros_like(f.narrow(dim, 0, 1))
                    dif = torch.diff(f, dim=dim, prepend=edge) if kind == "e" else torch.diff(f, dim=dim, append=edge)
                    inv, b, a = self.prof[kind, axis]
                    q = 6 + 2 * (base + c) + t
                    s[q] = b * s[q] + a * dif
                    part = (dif * inv + s[q]) * (sign if kind == "e" else -sign)
                    total = part if total is None else total + part
                new.append(self.ca[base + c] * s[base + c] + self.cb[base + c] * total)
            if kind == "e":
                for box, cj, wave in self.inject:
                    if m < len(wave):
                        add = torch.zeros_like(new[2])
                        add[box] = cj * wave[m]
                        new[2] = new[2] + add
            s[base:base + 3] = new
        return s


def _exact_run(sc, seed, steps, device, with_fields=True):
    ex = _Exact(sc, device)
    f = [None] * 6
    if with_fields:
        gen_device = "cuda" if torch.cuda.is_available() else "cpu"
        for c, v in _start_fields(sc.nx, sc.ny, sc.nz, seed, gen_device):
            f[c] = v.to(device=device, dtype=torch.float64)
    s = ex.start(f if with_fields else None)
    rows = torch.zeros((steps, len(sc.probes)), dtype=torch.float64, device=device)
    for m in range(steps):
        s = ex.step(s, m)
        for q, p in enumerate(sc.probes):
            rows[m, q] = s[p.component][p.k, p.j, p.i]
    return rows, s[:6]


def _exact_marching(case, seed, device):
    a = _microstrip(case, seed)
    X, Y, Z, P, A, W = (case[q] for q in ("X", "Y", "Z", "pml", "air", "width"))
    o = P + A
    s0, s1 = X // 2 - W // 2, X // 2 - W // 2 + W
    p0, p1, pj0, pj1, vj = X // 5, X - X // 5, Y // 2, Y - Y // 8, Y // 6
    steps = case["steps"]
    g = lambda name: float(np.float32(a[name]))  # noqa: E731
    t = np.arange(steps) * g("dt") - g("t_0")
    wave = g("source_amp") * np.exp(-(t / g("tau")) ** 2)
    mats = [S.Material(), S.Material(eps_r=a["brick_eps_r_x"][0], sigma_e=4e-4)]
    sc = S.Scenario("microstrip", X + 2 * o, Y + 2 * o, Z + 2 * o, g("dx"), g("dy"), g("dz"), g("dt"), (P,) * 6, steps, mats,
                    [S.Brick((o, o, o, o + X, o + Y, o + 3), 1)],
                    [S.LumpedSource((o + s0, o, o, o + s1, o, o + 3), 50.0, wave)],
                    [S.Resistor((o + p1, o + pj1, o, o + p1, o + pj1, o + 3), 50.0)] if case["resistor"] else [])
    edges = []
    for i0, j0, i1, j1, k in ((0, 0, X, Y, 0), (s0, 0, s1, pj0, 3), (p0, pj0, p1, pj1, 3)):
        edges.append((0, o + i0, o + j0, o + i1 - 1, o + j1, o + k, 1e10))
        edges.append((1, o + i0, o + j0, o + i1, o + j1 - 1, o + k, 1e10))
    ex = _Exact(sc, device, edges=edges)
    V = torch.zeros(steps, dtype=torch.float64, device=device)
    cur = torch.zeros(steps, dtype=torch.float64, device=device)
    s = ex.start()
    dx, dy, dz = ex.d
    i0, i1, j = o + s0, o + s1, o + vj
    zlo, ze = o + (0 if case["current"] == 3 else 3), o + 3
    for m in range(steps):
        s = ex.step(s, m)
        V[m] = -dz / (i1 - i0 + 1) * s[EZ][o:o + 3, j, i0:i1 + 1].sum()
        if case["current"] == 2:
            cur[m] = (dz * (s[HZ][zlo:ze + 1, j - 1, i0 - 1].sum() - s[HZ][zlo:ze + 1, j - 1, i1].sum())
                      + dx * (s[HX][ze, j - 1, i0:i1 + 1].sum() - s[HX][zlo - 1, j - 1, i0:i1 + 1].sum()))
        else:
            k = ze - 1
            cur[m] = (dy * (s[HY][k, j, i1] - s[HY][k, j, i0 - 1])
                      + dx * (s[HX][k, j - 1, i0:i1 + 1].sum() - s[HX][k, j, i0:i1 + 1].sum()))
    cur[:-1] = (cur[:-1] + cur[1:]) / 2
    cur[-1] = (cur[-1] + cur[-2]) / 2
    return [V.cpu().numpy(), cur.cpu().numpy()]


def _exact_adjoint(case, seed, device):
    sc, box, eps, probe = _design(case, seed)
    e = torch.tensor(eps.astype(np.float64), device=device, requires_grad=True)
    ex = _Exact(sc, device, design=(box, e))
    s = ex.start()
    J = torch.zeros((), dtype=torch.float64, device=device)

    def segment(m0, m1, J, *s):
        for m in range(m0, m1):
            s = ex.step(s, m)
            J = J + ex.dt * s[EZ][probe[2], probe[1], probe[0]] ** 2
        return (J, *s)

    for m0 in range(0, case["steps"], 8):
        J, *s = torch.utils.checkpoint.checkpoint(segment, m0, min(m0 + 8, case["steps"]), J, *s, use_reentrant=False)
    J.backward()
    return [float(J.detach()), e.grad.cpu().numpy()]


def exact(case, seed):
    """What run() returns for the first pass on prepare(case, seed), in 64 bits; None where it would
    take long or not fit."""
    gpu = torch.cuda.is_available()
    device = "cuda" if gpu else "cpu"
    kind = case["kind"]
    if kind in ("run", "job"):
        cells = case["nx"] * case["ny"] * case["nz"]
        if cells > 1.5e8 or cells * case["steps"] > (4e9 if gpu else 3e6):
            return None
        rows, f = _exact_run(_scenario(case, seed), seed, case["steps"], device, kind == "run")
        return [rows.cpu().numpy(), torch.stack(f)]
    if kind == "batch":
        if not gpu:
            return None
        parts = []
        for q, sc in enumerate(_batch_scenarios(case, seed)):
            parts += [v.reshape(-1) for v in _exact_run(sc, 7919 * seed + q, case["steps"], device)[1]]
        return torch.cat(parts)
    if kind == "adjoint":
        if not gpu and case["n"] ** 3 * case["steps"] > 1e7:
            return None
        return _exact_adjoint(case, seed, device)
    if not gpu:
        return None
    return _exact_marching(case, seed, device)
