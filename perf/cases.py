"""Performance cases of the Gross-Pitaevskii stepper: the calls its users make, at the sizes
they make them, from the smallest to the largest, with the inputs of each made from a seed.

A case is a dict of plain values: the kind of call ("what"), the lattice and its dimensions in
block cells, the spinor's components, the scheme and the storage precision, and how many steps
one call takes.  `prepare` builds the steppers and puts seeded states into their buffers, `run`
makes one pass through the public entry points, `exact` gives the same pass in 64 bits, written
out with torch on the stencil tables, and `work` the bytes and operations the pass needs.

The states are what a run meets some way into an evolution: a Thomas-Fermi cloud of c0 = 2000 in
a trap of omega = 1, displaced from the trap's centre, with a phase gradient and (spinors) a spin
texture, and 1e-3 noise.  Units and field ramps are those of the reference programs' set-ups.
"""
import json
import math
import os
import random

import numpy as np
import torch

from spacetime_gb300 import capi
from spacetime_gb300.adjoint import FinalStateObservables
from spacetime_gb300.batch import Batch
from spacetime_gb300.stepper import Stepper

C0, SIGMA, DT_HYPER, TRAP_OFFSET = 2000.0, 0.00225, 2e-5, 100.0
SCHEMES = {"parabolic": capi.SCHEME_PARABOLIC, "hyperbolic": capi.SCHEME_HYPERBOLIC, "split": capi.SCHEME_SPLIT}
EDGE_LATTICES = ("cube", "bcc", "bcc227", "c15")  # those that carry dual-edge tables
LATTICES = EDGE_LATTICES + ("fcc", "a15", "z")


def case(what, lattice, dims, components, steps, scheme="parabolic", bits=32, name=None, **more):
    c = {"what": what, "lattice": lattice, "x": dims[0], "y": dims[1], "z": dims[2], "components": components,
         "steps": steps, "scheme": scheme, "bits": bits, **more}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # a host loop that advances a small spinor a few steps at a time and looks at it in between
        case("step", "bcc", (12, 12, 12), 3, 4, name="spin1-bcc-12"),
        # the scalar vortex run on 32^3 BCC cells, a hundred steps a call: every step fits in L2
        case("step", "bcc", (32, 32, 32), 1, 100, name="scalar-bcc-32"),
        # the scalar C15 program on a grid whose edges are odd
        case("step", "c15", (41, 37, 35), 1, 50, name="scalar-c15-41"),
        # the spin-1 monopole run: a hundred steps under a field ramp, then norm, energy and magnetisation
        case("step_observe", "bcc", (96, 96, 96), 3, 100, name="spin1-bcc-96"),
        # the spin-2 program on a ragged box
        case("step", "bcc", (61, 57, 66), 5, 40, name="spin2-bcc-61"),
        # the relativistic (psi and q) spin-2 program on C15
        case("step", "c15", (40, 40, 40), 5, 32, scheme="hyperbolic", name="hyper-spin2-c15-40"),
        # the relativistic scalar C15 program, real and imaginary parts half a step apart
        case("step", "c15", (36, 36, 36), 1, 32, scheme="split", name="split-c15-36"),
        # the ground state by imaginary time, with which every run begins
        case("itp", "bcc", (72, 72, 72), 3, 32, name="itp-spin1-bcc-72"),
        # what a run records at a save step: all observables and the integrated spin fields
        case("observe", "bcc", (64, 64, 64), 3, 1, name="observe-spin1-bcc-64"),
        # a whole run in double precision: state from the host, Euler start, steps, observables, state to the host
        case("host_run", "bcc", (40, 40, 40), 3, 40, bits=64, name="run-f64-spin1-bcc-40"),
        # one gradient of a field-ramp control problem: recorded forward run, reverse run
        case("adjoint", "bcc", (40, 40, 40), 3, 200, name="adjoint-spin1-bcc-40"),
        # an ensemble of uneven condensates, scalar and spin-1, on four lattices, stepped together
        case("ensemble", "mixed", (24, 24, 60), 3, 10, name="ensemble-24", members=24, mix=1),
    ]


def draw(rng):
    """One more case: the kinds of the listed ones over their whole range of sizes."""
    def loguniform(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def dims(lattice, sites):
        edge = (sites / tables(lattice)["V"]) ** (1 / 3)
        return tuple(max(2, round(edge * rng.uniform(0.85, 1.15))) for _ in range(3))

    while True:
        what = rng.choices(("step", "step_observe", "itp", "observe", "host_run", "adjoint", "ensemble"),
                           (9, 3, 3, 2, 2, 2, 2))[0]
        sites, steps = loguniform(2e4, 1.2e7), round(loguniform(1, 100))
        bits, scheme = rng.choice((32, 32, 32, 64)), "parabolic"
        components = rng.choice((1, 3, 3, 5))
        lattice = rng.choice(("bcc", "bcc", "bcc") + LATTICES)
        if what == "step":
            scheme = rng.choice(("parabolic", "parabolic", "parabolic", "hyperbolic", "hyperbolic", "split"))
        if what == "itp" and lattice in EDGE_LATTICES and rng.random() < 0.3:
            scheme = "hyperbolic"
        if scheme != "parabolic" and lattice not in EDGE_LATTICES:
            lattice = rng.choice(("bcc", "c15"))
        if scheme == "split":
            components = 1
        if what == "ensemble":
            lo = round(loguniform(8, 40))
            c = case(what, "mixed", (lo, lo, lo + rng.randrange(1, 25)), 3, round(loguniform(2, 20)),
                     members=round(loguniform(2, 24)), mix=rng.randrange(1 << 20))
        elif what == "adjoint":
            c = case(what, "bcc", dims("bcc", loguniform(2e4, 1.2e6)), 3, round(loguniform(20, 200)))
        elif what == "host_run":
            c = case(what, lattice, dims(lattice, loguniform(2e4, 1.5e6)), components, round(loguniform(5, 40)), bits=64)
        else:
            c = case(what, lattice, dims(lattice, sites), components, 1 if what == "observe" else steps, scheme, bits)
        if work(c)["bytes"] <= 70e9 and work(c)["flops"] * (40 if c["bits"] == 64 else 1) <= 1.5e12:
            return c


# ------------------------------------------------------------------ lattices and parameters

_tables = {}


def tables(lattice):
    """The lattice's tables as the package ships them, as arrays (mixed rows padded with zero weights)."""
    if lattice not in _tables:
        with open(os.path.join(capi.LATTICE_DIR, lattice + ".json")) as f:
            d = json.load(f)
        V, ptr, st = int(d["nodes"]), d["row_ptr"], np.array(d["stencil"], dtype=np.float64)
        deg = max(ptr[i + 1] - ptr[i] for i in range(V))
        offset, node, hodge = np.zeros((V, deg, 3), int), np.tile(np.arange(V)[:, None], (1, deg)), np.zeros((V, deg))
        for i in range(V):
            for k, f in enumerate(range(ptr[i], ptr[i + 1])):
                offset[i, k], node[i, k], hodge[i, k] = st[f, :3].astype(int), int(st[f, 3]), st[f, 4]
        t = {"V": V, "entries": len(st), "bw": np.array(d["block_width"], float), "volume": float(d["volume"]),
             "pos": np.array(d["pos"], float).reshape(V, 3), "offset": offset, "node": node, "hodge": hodge, "E": 0}
        if "edges" in d:
            ed, inc = np.array(d["edges"], int), np.array(d["incidence"], float).reshape(V, -1, 5)
            t.update(E=len(ed), e_from=ed[:, 0], e_offset=ed[:, 1:4], e_to=ed[:, 4], i_offset=inc[..., :3].astype(int),
                     i_edge=inc[..., 3].astype(int), i_hodge=inc[..., 4])
        _tables[lattice] = t
    return _tables[lattice]


def setup(c):
    """The physics of a case: plain numbers, for the parameters and for `exact`."""
    t = tables(c["lattice"])
    dims = (c["x"], c["y"], c["z"])
    bs = 16.0 / (max(t["bw"][i] * dims[i] for i in range(3)))
    half = [0.5 * bs * t["bw"][i] * dims[i] for i in range(3)]
    spin = {1: (0.0, 0.0), 3: (-50.0, 0.0), 5: (-20.0, 40.0)}[c["components"]]
    # a tenth of the inverse of the largest local energy: kinetic bound, trap and offset, interaction
    energy = np.abs(t["hodge"]).sum(1).max() / bs ** 2 + 0.5 * sum(h * h for h in half) + TRAP_OFFSET + 15.0
    dt = 0.1 / energy if c["scheme"] == "parabolic" else DT_HYPER
    return dict(dims=dims, bs=bs, p0=[-h for h in half], dt=dt, lam=(1.0, 0.9, 1.1), c0=C0, c2=spin[0], c4=spin[1],
                ramp=4000 * dt)


def params(c, lattice):
    s = setup(c)
    return capi.make_params(components=c["components"], scheme=SCHEMES[c["scheme"]],
                            precision=capi.FP64 if c["bits"] == 64 else capi.FP32, dims=s["dims"], block_scale=s["bs"],
                            p0=s["p0"], dt=s["dt"], trap_lambda=s["lam"], trap_offset=TRAP_OFFSET, c0=s["c0"],
                            c2=s["c2"], c4=s["c4"], sigma=SIGMA if c["scheme"] != "parabolic" else 0.0, lattice=lattice)


BXY, BZ, BQ = (0.1, -0.05), 0.5, 0.2  # the bias field is (BXY, from BZ to -BZ over 4000 steps); BQ the gradient


def ramp(s):
    return capi.make_ramp(bq_segments=[(BQ, 1e9, capi.RAMP_CONSTANT)],
                          bb_segments=[((*BXY, BZ), 0.0, capi.RAMP_CONSTANT), ((*BXY, -BZ), s["ramp"], capi.RAMP_LINEAR),
                                       ((*BXY, -BZ), 1e9, capi.RAMP_CONSTANT)])


def fields_at(s, t):
    bz = BZ - 2 * BZ * min(t / s["ramp"], 1.0)
    return torch.tensor([BQ, *BXY, bz], dtype=torch.float64, device="cuda")


# ------------------------------------------------------------------ states


def positions(c):
    t, s = tables(c["lattice"]), setup(c)
    X, Y, Z = s["dims"]
    out = torch.empty((Z, Y, X, t["V"], 3), dtype=torch.float64, device="cuda")
    for i, n in enumerate((X, Y, Z)):
        shape = [1, 1, 1, 1]
        shape[2 - i] = n
        cell = torch.arange(n, dtype=torch.float64, device="cuda").reshape(shape) * float(t["bw"][i])
        out[..., i] = s["p0"][i] + s["bs"] * (cell + torch.tensor(t["pos"][:, i], device="cuda"))
    return out


ZETA = {1: (1.0,), 3: (0.62, 0.66, 0.42), 5: (0.55, 0.3, 0.45, 0.5, 0.4)}


def seeded_state(c, seed):
    """A normalised state of the case's grid, rounded to its storage precision: (Z, Y, X, V, C, 2), 64 bits."""
    t, s, C = tables(c["lattice"]), setup(c), c["components"]
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = positions(c)
    shift = [rng.uniform(0.2, 0.5) * rng.choice((-1, 1)) for _ in range(3)]
    lam = s["lam"]
    mu = 0.5 * (15 * s["c0"] * lam[0] * lam[1] * lam[2] / (4 * math.pi)) ** 0.4
    amp = torch.zeros(r.shape[:4], dtype=torch.float64, device="cuda")
    for i in range(3):
        amp += 0.5 * (lam[i] * (r[..., i] - shift[i])) ** 2
    amp = ((mu - amp).clamp_(min=0) / s["c0"]).sqrt_()
    psi = torch.empty((*r.shape[:4], C, 2), dtype=torch.float64, device="cuda")
    noise = 1e-3 * math.sqrt(mu / s["c0"])
    for m in range(C):
        k = [rng.uniform(-0.3, 0.3) for _ in range(3)]
        phase = k[0] * r[..., 0] + k[1] * r[..., 1] + k[2] * r[..., 2]
        if C == 1:  # a straight vortex along z
            phase += torch.atan2(r[..., 1] - shift[1], r[..., 0] - shift[0])
        zeta = ZETA[C][m] * rng.uniform(0.9, 1.1)
        for part, f in enumerate((torch.cos, torch.sin)):
            psi[..., m, part] = zeta * amp * f(phase) + noise * torch.randn(amp.shape, generator=gen, dtype=torch.float64, device="cuda")
    psi *= 1 / math.sqrt(float(psi.square().sum()) * s["bs"] ** 3 * t["volume"])
    return psi.float().double() if c["bits"] == 32 else psi


class _Memory:
    """A stepper's buffer for torch, which keeps this object, and with it the stepper, as long as the tensor lives."""

    def __init__(self, owner, **interface):
        self.owner = owner
        self.__cuda_array_interface__ = interface


def view(stepper, slot):
    """A slot's interior as a torch tensor over the stepper's own memory: (Z, Y, X, V or E, C, 2)."""
    p, cell = stepper.buffer(slot)
    par = stepper.params
    bits = 8 if par.precision == capi.FP64 else 4
    items = stepper.lattice.edges if slot in (capi.Q_EVEN, capi.Q_ODD) else stepper.lattice.nodes
    C = par.components
    return torch.as_tensor(_Memory(stepper, shape=(par.dims[2], par.dims[1], par.dims[0], items, C, 2),
                                   typestr="<f%d" % bits, data=(p.ptr, False), version=3,
                                   strides=(p.slice_pitch, p.pitch, cell, 2 * C * bits, 2 * bits, bits)), device="cuda")


def padded(psi):
    out = torch.zeros((psi.shape[0] + 2, psi.shape[1] + 2, psi.shape[2] + 2, *psi.shape[3:]), dtype=psi.dtype, device=psi.device)
    out[1:-1, 1:-1, 1:-1] = psi
    return out


def pinned(psi):
    """A state as a pinned host array in the file layout, halo included."""
    host = torch.empty([psi.shape[0] + 2, psi.shape[1] + 2, psi.shape[2] + 2, *psi.shape[3:]], dtype=torch.float64, pin_memory=True)
    host.copy_(padded(psi))
    return host.numpy()


# ------------------------------------------------------------------ one pass


def new_stepper(c, seed, start=True):
    s = Stepper(c["lattice"], params(c, capi.Lattice(c["lattice"])))
    slot = capi.PSI_EVEN if c["scheme"] == "split" else capi.PSI_ODD
    view(s, slot).copy_(seeded_state(c, seed))
    torch.cuda.synchronize()
    if c["components"] > 1:
        s.set_ramp(ramp(setup(c)), 0.0)
    if start:
        s.start()
    return s


def ensemble_members(c):
    rng = random.Random(c["mix"])
    out = []
    for _ in range(c["members"]):
        lattice, components = rng.choice(("bcc", "fcc", "a15", "c15")), rng.choice((1, 3))
        edge = rng.randint(c["x"], c["z"])
        # the same physical box with fewer cells of the lattices that have more nodes a cell
        edge = max(2, round(edge * (12 / tables(lattice)["V"]) ** (1 / 3)))
        out.append(case("step", lattice, (edge, edge, edge), components, c["steps"]))
    return out


def target_seed(seed):
    return 7919 * seed + 1


ADJOINT_SEED = (0.7, -0.4, 0.2, -0.1, 0.3)  # dL/d(overlap, magnetisation) of the control problem's loss


def adjoint_fields(c, seed):
    """A field schedule of a control problem: (steps, 4), smooth, as 32-bit parameters."""
    rng = random.Random(seed)
    s = np.arange(c["steps"]) / max(c["steps"] - 1, 1)
    f = np.stack([sum(rng.uniform(-0.5, 0.5) * np.cos(k * math.pi * s) for k in range(4)) for _ in range(4)], axis=1)
    return f.astype(np.float32)


def prepare(c, seed):
    if c["what"] == "ensemble":
        members = [new_stepper(m, seed + 101 * k) for k, m in enumerate(ensemble_members(c))]
        return {"case": c, "members": members, "batch": Batch(members)}
    state = {"case": c, "stepper": new_stepper(c, seed, start=c["what"] in ("step", "step_observe"))}
    s = state["stepper"]
    if c["what"] == "host_run":
        state["host"] = pinned(seeded_state(c, seed))
        state["result"] = torch.empty(state["host"].shape, dtype=torch.float64, pin_memory=True).numpy()
    if c["what"] == "adjoint":
        state["initial"] = view(s, capi.PSI_ODD).clone()
        state["target"] = padded(seeded_state(c, target_seed(seed))).cpu().numpy()
        state["fields"] = torch.from_numpy(adjoint_fields(c, seed))
    return state


def slots(s, c):
    """The leapfrog's pair of states (newest first), with q where the scheme has it."""
    if c["scheme"] == "split":
        return {"psi": view(s, capi.PSI_EVEN), "q": view(s, capi.Q_EVEN)}
    cur = s.current
    old = capi.PSI_ODD if cur == capi.PSI_EVEN else capi.PSI_EVEN
    out = {"psi": view(s, cur), "psi_before": view(s, old)}
    if c["scheme"] == "hyperbolic":
        q = {capi.PSI_EVEN: capi.Q_EVEN, capi.PSI_ODD: capi.Q_ODD}
        out.update(q=view(s, q[cur]), q_before=view(s, q[old]))
    return out


def numbers(o, C):
    """The observables that mean something for C components (a scalar has no spin)."""
    keep = ("norm", "energy", "h_expect", "com", "max_abs") + (("magnetization", "spin_norm") if C > 1 else ())
    return {k: o[k] for k in keep}


def run(state):
    c = state["case"]
    what, C = c["what"], c["components"]
    if what == "ensemble":
        state["batch"].step(c["steps"])
        return [view(s, s.current) for s in state["members"]]
    s = state["stepper"]
    if what == "step":
        s.step(c["steps"])
        return slots(s, c)
    if what == "step_observe":
        return {"observed": numbers(s.step_observe(c["steps"]), C), **slots(s, c)}
    if what == "itp":
        mu = s.itp(c["steps"])
        return {"mu": mu, "hpsi": view(s, capi.HPSI), **slots(s, c)}
    if what == "observe":
        out = {"observed": numbers(s.observe(s.current, 0.25 * setup(c)["ramp"]), C),
               "density": s.node_fields_reduce(s.current, capi.FIELD_DENSITY).tolist()}
        if C > 1:
            out["spin"] = s.node_fields_reduce(s.current, capi.FIELD_SPIN).tolist()
        return out
    if what == "host_run":
        s.upload(capi.PSI_ODD, state["host"])
        if C > 1:
            s.set_ramp(ramp(setup(c)), 0.0)
        s.start()
        s.step(c["steps"])
        observed = s.observe(s.current, c["steps"] * s.params.dt)
        return {"observed": numbers(observed, C), "result": s.download(s.current, state["result"])}
    if what == "adjoint":
        fields = state["fields"].clone().requires_grad_(True)
        out = FinalStateObservables.apply(fields, s, lambda: view(s, capi.PSI_ODD).copy_(state["initial"]), state["target"])
        out.backward(torch.tensor(ADJOINT_SEED, dtype=out.dtype))
        return {"final": out.tolist(), "gradient": fields.grad}
    raise ValueError(what)


# ------------------------------------------------------------------ what a pass needs


def work(c):
    if c["what"] == "ensemble":
        parts = [work(m) for m in ensemble_members(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    t, C, b, n = tables(c["lattice"]), c["components"], c["bits"] // 8, c["steps"]
    sites = c["x"] * c["y"] * c["z"] * t["V"]
    record = 2 * C * b  # one read or one write of psi at a site
    local = {1: 22, 3: 110, 5: 260}[C]
    flops = sites * (4 * C * t["entries"] / t["V"] + 2 * C + local + 4 * C)
    edges = t["E"] / t["V"]
    if c["scheme"] != "parabolic":
        flops += sites * edges * 10 * C
    if c["what"] == "observe":  # each call reads the state once
        return {"bytes": sites * record * (3 if C > 1 else 2), "flops": flops + sites * 80}
    step = 3 * record * (1 + (edges if c["scheme"] != "parabolic" else 0))  # read prev, read and write next
    if c["what"] == "itp":  # read prev, write next; H psi once
        both = 2 * record * (1 + (edges if c["scheme"] != "parabolic" else 0))
        return {"bytes": sites * (both * n + record), "flops": n * flops}
    if c["what"] == "host_run":  # the state in and out once, the Euler start, the steps, the observables
        host = 8 * 2 * C * (c["x"] + 2) * (c["y"] + 2) * (c["z"] + 2) * t["V"]
        return {"bytes": 2 * host + sites * (2 * record + step * n + record), "flops": (n + 2) * flops}
    if c["what"] == "adjoint":  # forward step; reverse step: u, lambda read, the older lambda read and written
        return {"bytes": sites * n * (step + 4 * record), "flops": 3 * n * flops}
    return {"bytes": sites * step * n, "flops": n * flops}


# ------------------------------------------------------------------ the same in 64 bits


class Grid:
    """A case's stencil as gathers over flat arrays: `pad` holds the cells with their zero halo."""

    def __init__(self, c):
        t, s = tables(c["lattice"]), setup(c)
        self.c, self.s, self.t, self.V, self.E = c, s, t, t["V"], t["E"]
        X, Y, Z = s["dims"]
        self.shape = (Z, Y, X)
        z, y, x = torch.meshgrid(*(torch.arange(n, device="cuda") for n in (Z, Y, X)), indexing="ij")
        cell = lambda d: (((z + 1 + int(d[2])) * (Y + 2) + y + 1 + int(d[1])) * (X + 2) + x + 1 + int(d[0])).reshape(-1, 1)  # noqa: E731

        def gather(offsets, items, per):
            return torch.cat([cell(o) * per + int(i) for o, i in zip(offsets, items)], dim=1).reshape(-1)

        up = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
        cells = X * Y * Z
        self.near = [gather(t["offset"][:, k], t["node"][:, k], self.V) for k in range(t["hodge"].shape[1])]
        self.weight = [up(-0.5 * t["hodge"][:, k] / s["bs"] ** 2).repeat(cells)[:, None] for k in range(len(self.near))]
        if c["scheme"] != "parabolic":
            self.inc = [gather(t["i_offset"][:, k], t["i_edge"][:, k], self.E) for k in range(t["i_hodge"].shape[1])]
            self.inc_weight = [up(-0.5 * t["i_hodge"][:, k] / s["bs"] ** 2).repeat(cells)[:, None] for k in range(len(self.inc))]
            self.e_from = gather([(0, 0, 0)] * self.E, t["e_from"], self.V)
            self.e_to = gather(t["e_offset"], t["e_to"], self.V)
        self.r = positions(c).reshape(-1, 3)
        lam = up(s["lam"])
        self.trap = 0.5 * ((self.r * lam) ** 2).sum(1, keepdim=True) + TRAP_OFFSET

    def pad(self, v):
        v = v.reshape(*self.shape, -1, v.shape[-1])
        out = torch.zeros((self.shape[0] + 2, self.shape[1] + 2, self.shape[2] + 2, *v.shape[3:]), dtype=v.dtype, device="cuda")
        out[1:-1, 1:-1, 1:-1] = v
        return out.reshape(-1, v.shape[-1])

    def kinetic(self, psi):
        p = self.pad(psi)
        out = 0
        for i, w in zip(self.near, self.weight):
            out = out + w * (p[i] - psi)
        return out

    def d0(self, psi):
        p = self.pad(psi)
        return p[self.e_to] - p[self.e_from]

    def d1(self, q):
        p = self.pad(q)
        return sum(w * p[i] for i, w in zip(self.inc, self.inc_weight))

    def field(self, f):
        """The magnetic field at the nodes for f = (Bq, Bx, By, Bz)."""
        x, y, z = self.r[:, :1], self.r[:, 1:2], self.r[:, 2:]
        return f[0] * x + f[1], f[0] * y + f[2], -2 * f[0] * z + f[3]

    def zeeman(self, B, psi):
        """(B.F) psi for spin 1."""
        bxy = torch.complex(*torch.broadcast_tensors(B[0], B[1])) / math.sqrt(2)
        u, v, w = psi[:, :1], psi[:, 1:2], psi[:, 2:]
        return torch.cat([B[2] * u + bxy.conj() * v, bxy * u + bxy.conj() * w, bxy * v - B[2] * w], dim=1)

    def spin(self, psi):
        """<F> of the unnormalised spinor."""
        a = psi.abs() ** 2
        if psi.shape[1] == 3:
            m = math.sqrt(2) * (psi[:, 0].conj() * psi[:, 1] + psi[:, 1].conj() * psi[:, 2])
            fz = a[:, 0] - a[:, 2]
        else:
            m = 2 * (psi[:, 0].conj() * psi[:, 1] + psi[:, 3].conj() * psi[:, 4]) + \
                math.sqrt(6) * (psi[:, 1].conj() * psi[:, 2] + psi[:, 2].conj() * psi[:, 3])
            fz = 2 * a[:, 0] + a[:, 1] - a[:, 3] - 2 * a[:, 4]
        return m.real[:, None], m.imag[:, None], fz[:, None]

    def potential(self, psi):
        return self.trap + self.s["c0"] * (psi.abs() ** 2).sum(1, keepdim=True)

    def spin_part(self, psi, f):
        """The spin interaction and the Zeeman term; f None leaves the external field out."""
        C, s = psi.shape[1], self.s
        if C == 1:
            return 0 * psi
        B = self.field(f) if f is not None else (0 * self.trap,) * 3
        if C == 3:
            return self.zeeman(tuple(b + s["c2"] * m for b, m in zip(B, self.spin(psi))), psi)
        a = psi.abs() ** 2
        s2, s1, s0, t1, t2 = (psi[:, k:k + 1] for k in range(5))
        n = [a[:, k:k + 1] for k in range(5)]
        c2, c4 = s["c2"], s["c4"]
        fz = c2 * (2 * n[0] + n[1] - n[3] - 2 * n[4])
        den = c2 * (2 * (s2 * s1.conj() + t1 * t2.conj()) + math.sqrt(6) * (s1 * s0.conj() + s0 * t1.conj())) - torch.complex(B[0], -B[1])
        c12, c45 = den - 0.4 * c4 * t1 * t2.conj(), den - 0.4 * c4 * s2 * s1.conj()
        c13, c35 = 0.2 * c4 * s0 * t2.conj(), 0.2 * c4 * s2 * s0.conj()
        c23, c34 = math.sqrt(1.5) * den - 0.2 * c4 * s0 * t1.conj(), math.sqrt(1.5) * den - 0.2 * c4 * s1 * s0.conj()
        return torch.cat([(2 * fz + 0.4 * c4 * n[4] - 2 * B[2]) * s2 + c12 * s1 + c13 * s0,
                          (fz + 0.4 * c4 * n[3] - B[2]) * s1 + c12.conj() * s2 + c23 * s0,
                          0.2 * c4 * n[2] * s0 + c13.conj() * s2 + c35 * t2 + c34 * t1 + c23.conj() * s1,
                          (-fz + 0.4 * c4 * n[1] + B[2]) * t1 + c34.conj() * s0 + c45 * t2,
                          (-2 * fz + 0.4 * c4 * n[0] + 2 * B[2]) * t2 + c35.conj() * s0 + c45.conj() * t1], dim=1)

    def h(self, psi, f):
        return self.kinetic(psi) + self.potential(psi) * psi + self.spin_part(psi, f)

    def observables(self, psi, f, C):
        s = self.s
        dv = s["bs"] ** 3 * self.t["volume"]
        total = lambda v: float(v.sum()) * dv  # noqa: E731
        rho = (psi.abs() ** 2).sum(1, keepdim=True)
        h = total((psi.conj() * self.h(psi, f)).real)
        interaction = total(s["c0"] * rho ** 2) + (total((psi.conj() * self.spin_part(psi, None)).real) if C > 1 else 0)
        out = {"norm": total(rho), "energy": h - 0.5 * interaction, "h_expect": h,
               "com": [total(rho * self.r[:, i:i + 1]) for i in range(3)], "max_abs": float(psi.abs().max())}
        if C > 1:
            m = self.spin(psi)
            out.update(magnetization=[total(v) for v in m], spin_norm=total((m[0] ** 2 + m[1] ** 2 + m[2] ** 2).sqrt()))
        return out

    def back(self, v):
        """A flat complex state in the outputs' layout."""
        return torch.view_as_real(v.reshape(*self.shape, -1, v.shape[-1]))


def _exact_steps(c, seed):
    """The start and the steps of a pass: (grid, newest, older, time of the last step, q, older q)."""
    g, s, n = Grid(c), setup(c), c["steps"]
    dt = s["dt"]
    old = torch.view_as_complex(seeded_state(c, seed)).reshape(-1, c["components"])
    if c["scheme"] == "split":
        dts = dt / SIGMA
        k = dts / (dt - dts)
        R, I = old.real.clone(), old.imag.clone()  # noqa: E741
        qr = k * g.d0(R)
        qi = torch.zeros_like(qr)
        for _ in range(n):
            I, qi = I - dt * ((g.trap + s["c0"] * (R ** 2 + I ** 2)) * R - g.d1(qr)), qi + dts * (qr + g.d0(R))  # noqa: E741
            R, qr = R + dt * ((g.trap + s["c0"] * (R ** 2 + I ** 2)) * I - g.d1(qi)), qr - dts * (qi + g.d0(I))
        return g, torch.complex(R, I), None, n * dt, torch.complex(qr, qi), None
    spinor = c["components"] > 1
    f = lambda t: fields_at(s, t) if spinor else torch.zeros(4, dtype=torch.float64, device="cuda")  # noqa: E731
    if c["scheme"] == "parabolic":
        new = old - 1j * dt * g.h(old, f(0.0))
        for k in range(1, n + 1):
            old, new = new, old - 2j * dt * g.h(new, f(k * dt))
        return g, new, old, n * dt, None, None
    q_old = g.d0(old)
    new = old - 1j * dt * (g.d1(q_old) + g.potential(old) * old + g.spin_part(old, f(0.0)))
    q_new = g.d0(new)
    for k in range(1, n + 1):
        pot = g.potential(new)
        h = -(1 + SIGMA * pot) * g.d1(q_new) + pot * new + g.spin_part(new, f(k * dt))
        old, new, q_old, q_new = new, old - 2j * dt * h, q_new, q_old + 2j * dt / SIGMA * (q_new + g.d0(new))
    return g, new, old, n * dt, q_new, q_old


def _exact_pair(c, seed):
    g, new, old, t, q_new, q_old = _exact_steps(c, seed)
    out = {"psi": g.back(new)}
    if old is not None:
        out["psi_before"] = g.back(old)
    if q_new is not None:
        out["q"] = g.back(q_new)
    if q_old is not None:
        out["q_before"] = g.back(q_old)
    return g, new, old, t, out


def _exact_adjoint(c, seed):
    g, s, n = Grid(c), setup(c), c["steps"]
    dt, dv = s["dt"], s["bs"] ** 3 * g.t["volume"]
    fields = torch.from_numpy(adjoint_fields(c, seed)).double().cuda()
    target = torch.view_as_complex(seeded_state({**c, "bits": 32}, target_seed(seed))).reshape(-1, c["components"])
    u = [torch.view_as_complex(seeded_state(c, seed)).reshape(-1, c["components"])]
    for j in range(n):
        u.append((u[j - 1] if j else u[0]) - (2j if j else 1j) * dt * g.h(u[j], fields[j]))

    def final(v):
        m = g.spin(v)
        o = (target.conj() * v).sum()
        return torch.stack([o.real, o.imag, m[0].sum(), m[1].sum(), m[2].sum()]) * dv

    def pull(fn, point, f, cotangent):
        p, q = point.detach().requires_grad_(True), f.detach().requires_grad_(True)
        return torch.autograd.grad(fn(p, q), (p, q), cotangent)

    p = u[n].detach().requires_grad_(True)
    out = final(p)
    after, lam = torch.zeros_like(p), torch.autograd.grad(out, p, torch.tensor(ADJOINT_SEED, dtype=torch.float64, device="cuda"))[0]
    gradient = torch.zeros((n, 4), dtype=torch.float64)
    for j in range(n - 1, -1, -1):
        d, df = pull(lambda v, f: -(2j if j else 1j) * dt * g.h(v, f), u[j], fields[j], lam)
        gradient[j] = df.cpu()
        after, lam = lam, after + d
    return {"final": out.tolist(), "gradient": gradient}


def exact(c, seed):
    what, C = c["what"], c["components"]
    if what == "ensemble":
        out = []
        for k, m in enumerate(ensemble_members(c)):
            g, new, *_ = _exact_steps(m, seed + 101 * k)
            out.append(g.back(new))
        return out
    if what == "adjoint":
        return _exact_adjoint(c, seed)
    s = setup(c)
    if what == "observe":
        g = Grid(c)
        psi = torch.view_as_complex(seeded_state(c, seed)).reshape(-1, C)
        f = fields_at(s, 0.25 * s["ramp"]) if C > 1 else torch.zeros(4, dtype=torch.float64, device="cuda")
        o = g.observables(psi, f, C)
        # the integrated spin fields: sizes and z projection of the spinor over its density's root
        return {"observed": o, "density": [o["norm"]], **({"spin": None} if C > 1 else {})}
    if what == "itp":
        g, dt, dv = Grid(c), s["dt"], s["bs"] ** 3 * tables(c["lattice"])["volume"]
        new = torch.view_as_complex(seeded_state(c, seed)).reshape(-1, C)
        old = h = None
        hyper = c["scheme"] == "hyperbolic"
        q = q_old = torch.zeros((g.r.shape[0] // g.V * g.E, C), dtype=torch.complex128, device="cuda") if hyper else None
        for _ in range(c["steps"]):
            h = (g.d1(q) if hyper else g.kinetic(new)) + g.potential(new) * new + g.spin_part(new, None)
            if hyper:
                q_old, q = q, q - dt / SIGMA * (q - g.d0(new))
            old, new = new, new - dt * h
            new = new / ((new.abs() ** 2).sum() * dv).sqrt()
        out = {"mu": float((new.conj() * h).real.sum()) * dv, "hpsi": g.back(h), "psi": g.back(new), "psi_before": g.back(old)}
        if hyper:
            out.update(q=g.back(q), q_before=g.back(q_old))
        return out
    if what == "host_run":
        g, new, old, t, _, _ = _exact_steps(c, seed)
        f = fields_at(s, t) if C > 1 else torch.zeros(4, dtype=torch.float64, device="cuda")
        return {"observed": g.observables(new, f, C), "result": padded(g.back(new))}
    g, new, old, t, out = _exact_pair(c, seed)
    if what == "step_observe":
        f = fields_at(s, t) if C > 1 else torch.zeros(4, dtype=torch.float64, device="cuda")
        out["observed"] = g.observables(old, f, C)
    return out
