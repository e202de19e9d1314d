"""The work that programs have this package do, as timed cases.

Every case goes through the public Python API: fused time steps, the separate
operators of the reference's driver loop, batched ensembles, adjoints and the
FP64 MatlabPort front-end, on grids from 16x8x8 to 256x128x128, whole-tile
and ragged, with and without a nozzle.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call (on the GPU)
    run(state)          one pass; returns its outputs
    work(case)          bytes and operations a pass cannot do without
    exact(case, seed)   the outputs in 64 bits, from plain torch

The flows are smooth random ones (a run some steps in) and vortex rings; the
particles fill the region behind a nozzle or thin tori around the rings.
"""
import importlib
import math

import torch

import __graft_entry__

sf = __graft_entry__.load_package()
cfgs = importlib.import_module(sf.__name__ + ".configs")

HBAR = cfgs.HBAR
DT = cfgs.CONFIGS["C1"]["dt"]
# pencil lengths the library accepts (include/isf.h)
LENS = (8, 12, 16, 20, 24, 32, 40, 48, 50, 56, 64, 80, 96, 100, 112, 128, 160, 192, 200, 256, 384, 512)
MAX_CELLS = 256 * 128 * 128


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _case(name, kind, dims, size, **more):
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "lx": size[0], "ly": size[1], "lz": size[2]}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # the smallest call a program makes: one operator pair on the smallest grid of the tests (launch latency)
        _case("flow_16x8x8", "flow", (16, 8, 8), (4, 2, 2)),
        # the reference's jet at the interactive size: a fused step with 1000 births
        _case("jet_step_64x32x32", "step", (64, 32, 32), (4, 2, 2), jet=True, slots=100_000, emit=1000),
        # the reference's driver loop, operator by operator, at its test size
        _case("jet_loop_128x64x64", "loop", (128, 64, 64), (4, 2, 2), jet=True, slots=1 << 18, emit=2000),
        # the headline run: leapfrogging rings with 4M particles, no nozzle
        _case("rings_step_256x128x128", "step", (256, 128, 128), (10, 5, 5), jet=False, slots=1 << 22, emit=0),
        # the spectral step and the projection on ragged boxes (factors 5 and 7, ny != nz, partial tiles)
        _case("flow_200x112x100", "flow", (200, 112, 100), (6, 3, 3)),
        _case("project_100x50x56", "project", (100, 50, 56), (4, 2, 2)),
        # the velocity of a frame, read back by the caller
        _case("velocity_160x96x80", "velocity", (160, 96, 80), (5, 3, 3)),
        # a dye of 1M particles carried by a frozen jet, a ring buffer of births
        _case("advect_128x64x64", "advect", (128, 64, 64), (4, 2, 2), slots=1 << 20, emit=8192),
        # an ensemble of small jets of uneven sizes, a few steps between two looks at the state
        _case("batch_8_jets", "batch", (96, 48, 48), (6, 3, 3), sims=8, slots=32768, steps=4),
        # one reversed step, and a checkpointed gradient of the particle loss
        _case("adj_step_128x64x64", "adj_step", (128, 64, 64), (4, 2, 2), slots=1 << 18),
        _case("adj_gradient_64x32x32", "adj_gradient", (64, 32, 32), (4, 2, 2), slots=65536, init=2, steps=6, every=3),
        # the MatlabPort driver's field operators on its 64x32x32 jet grid, complex128 in and out
        _case("matlab_64x32x32", "matlab", (64, 32, 32), (4, 2, 2)),
    ]


def _draw_grid(rng, lo, hi):
    """A grid of lo..hi cells (log-uniform) with an x-long or cubic box; half of them with ny = nz."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.choice((1.0, 1.5, 2.0, 2.0, 3.0))
    want = (cells / aspect) ** (1 / 3)
    near = lambda v: min(LENS, key=lambda n: abs(math.log(n / v)) + 0.15 * rng.random())  # noqa: E731
    ny = near(want)
    nz = ny if rng.random() < 0.5 else near(want)
    nx = near(want * aspect)
    while nx * ny * nz > hi:
        nx = max(n for n in LENS if n < nx)
    per = rng.choice((16, 32))
    return (nx, ny, nz), tuple(max(1, round(n / per)) for n in (nx, ny, nz))


def draw(rng):
    kind = rng.choice(("flow", "project", "velocity", "step", "step", "loop", "advect", "batch", "adj_step",
                       "adj_gradient", "matlab"))
    if kind in ("flow", "project", "velocity"):
        return _case(None, kind, *_draw_grid(rng, 1024, MAX_CELLS))
    if kind == "step":
        dims, size = _draw_grid(rng, 16384, MAX_CELLS // 2)
        jet = rng.random() < 0.6
        slots = int(math.exp(rng.uniform(math.log(5000), math.log(1 << 21))))
        return _case(None, kind, dims, size, jet=jet, slots=slots, emit=slots // rng.randint(50, 200) if jet else 0)
    if kind == "loop":
        dims, size = _draw_grid(rng, 16384, MAX_CELLS // 8)
        slots = int(math.exp(rng.uniform(math.log(5000), math.log(1 << 19))))
        return _case(None, kind, dims, size, jet=True, slots=slots, emit=slots // rng.randint(50, 200))
    if kind == "advect":
        dims, size = _draw_grid(rng, 16384, MAX_CELLS // 2)
        slots = int(math.exp(rng.uniform(math.log(10000), math.log(1 << 22))))
        return _case(None, kind, dims, size, slots=slots, emit=slots // rng.randint(50, 200))
    if kind == "batch":
        return _case(None, kind, (96, 48, 48), (6, 3, 3), sims=rng.randint(3, 16), slots=rng.randint(4000, 65536),
                     steps=rng.randint(1, 8))
    if kind == "adj_step":
        dims, size = _draw_grid(rng, 16384, MAX_CELLS // 4)
        return _case(None, kind, dims, size, slots=int(math.exp(rng.uniform(math.log(5000), math.log(1 << 19)))))
    if kind == "adj_gradient":
        dims, size = _draw_grid(rng, 16384, MAX_CELLS // 32)
        steps = rng.randint(3, 8)
        return _case(None, kind, dims, size, slots=rng.randint(5000, 100_000), init=rng.randint(0, 3), steps=steps,
                     every=rng.randint(2, steps))
    return _case(None, "matlab", *_draw_grid(rng, 8192, MAX_CELLS // 4))


# ------------------------------------------------------------------- inputs
def _dims(c):
    return (c["nx"], c["ny"], c["nz"])


def _size(c):
    return (c["lx"], c["ly"], c["lz"])


def _rng(seed):
    return torch.Generator(device=_dev()).manual_seed(int(seed) * 7919 + 17)


def _uniform(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device=_dev(), dtype=torch.float64) * (hi - lo) + lo


def _axes(dims):
    """Cell coordinates in [0, 1) as (nz, ny, nx) broadcastable x, y, z."""
    nx, ny, nz = dims
    ar = lambda n: torch.arange(n, device=_dev(), dtype=torch.float64) / n  # noqa: E731
    return ar(nx)[None, None, :], ar(ny)[None, :, None], ar(nz)[:, None, None]


def _smooth(dims, g, modes=4):
    """A real periodic field of a few low Fourier modes (first harmonics only along an axis of under 32 cells)."""
    x, y, z = _axes(dims)
    top = torch.tensor([1 if n < 32 else 2 for n in dims], device=_dev())
    k = torch.randint(-2, 3, (modes, 3), generator=g, device=_dev())
    k = torch.minimum(torch.maximum(k, -top), top).tolist()
    ph = _uniform(g, modes, 0, 2 * math.pi).tolist()
    a = torch.randn(modes, generator=g, device=_dev(), dtype=torch.float64).tolist()
    f = torch.zeros(dims[::-1], device=_dev(), dtype=torch.float64)
    for m in range(modes):
        f += a[m] * torch.cos(2 * math.pi * (k[m][0] * x + k[m][1] * y + k[m][2] * z) + ph[m])
    return f


def _pack(p1, p2):
    n = torch.sqrt(p1.abs() ** 2 + p2.abs() ** 2)
    p1, p2 = p1 / n, p2 / n
    return torch.stack([p1.real, p1.imag, p2.real, p2.imag], dim=-1).to(torch.float32).contiguous()


def _smooth_psi(dims, g):
    """A normalised two-component psi with smooth phases and amplitudes."""
    th1, th2 = 0.8 * _smooth(dims, g), 0.8 * _smooth(dims, g)
    a1 = 1.0 + 0.2 * torch.tanh(_smooth(dims, g))
    a2 = 0.3 * (1.0 + 0.2 * torch.tanh(_smooth(dims, g)))
    return _pack(torch.polar(a1, th1), torch.polar(a2, th2))


def _rings(c):
    """(x centre, radius) of the two leapfrogging rings, scaled from the 10x5x5 box to the case's."""
    s = min(c["lx"] / 10, c["ly"] / 5, c["lz"] / 5)
    return [(x * s, r * s) for x, r in cfgs.CONFIGS["C3"]["rings"]], s


def _ring_psi(c, g):
    """The vortex-ring phase (a 2 pi jump across each ring's disc, spread over a slab) plus a weak smooth one."""
    dims, size = _dims(c), _size(c)
    x, y, z = (a * length for a, length in zip(_axes(dims), size))
    rings, s = _rings(c)
    delta = max(cfgs.CONFIGS["C3"]["delta"] * s, 3 * size[0] / dims[0])
    alpha = 0.05 * _smooth(dims, g)
    rho2 = (y - size[1] / 2) ** 2 + (z - size[2] / 2) ** 2
    for xc, r in rings:
        ax = -(x - xc)
        inside = rho2 < r * r
        alpha = alpha + torch.where(inside & (ax > 0) & (ax <= delta / 2), math.pi * (1 - 2 * ax / delta), 0.0)
        alpha = alpha + torch.where(inside & (ax <= 0) & (ax >= -delta / 2), -math.pi * (1 + 2 * ax / delta), 0.0)
    one = torch.ones_like(alpha)
    return _pack(torch.polar(one, alpha), torch.complex(0.01 * one, 0.0 * one))


def _cell_sorted(p, c):
    i = [(p[:, a] * (n / length)).long().clamp(0, n - 1) for a, (n, length) in enumerate(zip(_dims(c), _size(c)))]
    return p[torch.argsort(i[0] + c["nx"] * (i[1] + c["ny"] * i[2]))].to(torch.float32).contiguous()


def _ring_particles(c, g, n):
    """Thin tori around the rings, sorted by cell as the configurations seed them."""
    rings, s = _rings(c)
    which = torch.arange(n, device=_dev()) % len(rings)
    xc = torch.tensor([r[0] for r in rings], device=_dev(), dtype=torch.float64)[which]
    rad = torch.tensor([r[1] for r in rings], device=_dev(), dtype=torch.float64)[which]
    minor = cfgs.CONFIGS["C3"]["torus_minor"] * s * torch.sqrt(_uniform(g, n))
    th, phi = _uniform(g, n, 0, 2 * math.pi), _uniform(g, n, 0, 2 * math.pi)
    r = rad + minor * torch.cos(th)
    return _cell_sorted(torch.stack([xc + minor * torch.sin(th), c["ly"] / 2 + r * torch.cos(phi),
                                     c["lz"] / 2 + r * torch.sin(phi)], 1), c)


def _nozzle(c):
    """The reference's nozzle (4x2x2 box), scaled to the case's box."""
    n = cfgs.JET_NOZZLE
    s = min(c["lx"] / 4, c["ly"] / 2, c["lz"] / 2)
    kvec, omega = cfgs.jet_omega()
    f = lambda v: float(torch.tensor(v, dtype=torch.float32))  # noqa: E731
    return {"cen": (f(0.3 * c["lx"] / 4), f(n["cen"][1] * c["ly"] / 2), f(n["cen"][2] * c["lz"] / 2)),
            "len": f(n["len"] * c["lx"] / 4), "rad": f(n["rad"] * s), "kvec": kvec, "omega": omega}


def _jet_particles(c, g, n):
    """The stream behind the nozzle: births of the last steps, oldest furthest downstream."""
    noz = _nozzle(c)
    x = noz["cen"][0] + torch.linspace(0.5, 0.0, n, device=_dev(), dtype=torch.float64) * c["lx"]
    th, rho = _uniform(g, n, 0, 2 * math.pi), noz["rad"] * torch.sqrt(_uniform(g, n))
    return torch.stack([x + _uniform(g, n, -0.02, 0.02) * c["lx"], noz["cen"][1] + rho * torch.cos(th),
                        noz["cen"][2] + rho * torch.sin(th)], 1).to(torch.float32).contiguous()


def _jet_velocity(c):
    """A frozen jet (nz, ny, nx, 3): fast along x behind the nozzle, a slow swirl around it."""
    x, y, z = (a * length for a, length in zip(_axes(_dims(c)), _size(c)))
    noz = _nozzle(c)
    ry, rz = y - noz["cen"][1], z - noz["cen"][2]
    prof = torch.exp(-(ry ** 2 + rz ** 2) / noz["rad"] ** 2) + 0.0 * x
    return torch.stack([prof, -0.3 * rz * prof, 0.3 * ry * prof], dim=-1).to(torch.float32).contiguous()


def _fields(c, seed):
    """The case's input tensors, from the seed alone."""
    g, dims = _rng(seed), _dims(c)
    kind = c["kind"]
    if kind in ("flow", "project", "velocity", "matlab"):
        return {"psi": _smooth_psi(dims, g)}
    if kind in ("step", "loop"):
        if c["jet"]:
            return {"psi": _smooth_psi(dims, g), "parts": _jet_particles(c, g, c["slots"])}
        return {"psi": _ring_psi(c, g), "parts": _ring_particles(c, g, c["slots"])}
    if kind == "advect":
        return {"vel": _jet_velocity(c), "parts": _jet_particles(c, g, c["slots"])}
    if kind == "batch":
        out = {"sims": [], "psi": [], "parts": []}
        for i in range(c["sims"]):
            dims, size = cfgs.ENSEMBLE_GRIDS[i % len(cfgs.ENSEMBLE_GRIDS)]
            ci = {"nx": dims[0], "ny": dims[1], "nz": dims[2], "lx": size[0], "ly": size[1], "lz": size[2]}
            v = float(torch.tensor(0.5 + (i % 5) * 0.25, dtype=torch.float32))
            noz = _nozzle(ci)
            jet = dict(kvec=(float(torch.tensor(v / HBAR, dtype=torch.float32)), 0.0, 0.0),
                       omega=float(torch.tensor(v * v / (2 * HBAR), dtype=torch.float32)), cen=noz["cen"],
                       len=noz["len"], rad=noz["rad"], phase_mode=sf.PHASE_DOT, emit_mode=sf.EMIT_DISC,
                       emit_per_step=c["slots"] // 100, seed=int(seed) * 100 + i)
            out["sims"].append(dict(dims=dims, physical_size=size, hbar=HBAR, dt=DT, nslots=c["slots"], jet=jet))
            out["psi"].append(_smooth_psi(dims, g))
            out["parts"].append(_jet_particles(ci, g, c["slots"]))
        return out
    # the adjoints: a smooth state, particles in the box, cotangents / targets
    out = {"psi": _smooth_psi(dims, g)}
    box = torch.tensor(_size(c), device=_dev(), dtype=torch.float64)
    p = (0.1 + 0.8 * torch.rand((c["slots"], 3), generator=g, device=_dev(), dtype=torch.float64)) * box
    out["parts"] = _cell_sorted(p, c)
    if kind == "adj_step":
        out["psibar"] = torch.stack([_smooth(dims, g) for _ in range(4)], dim=-1).to(torch.float32).contiguous()
        out["partsbar"] = torch.randn((c["slots"], 3), generator=g, device=_dev(), dtype=torch.float32)
    else:
        out["targets"] = out["parts"] + 0.1 * torch.randn((c["slots"], 3), generator=g, device=_dev(),
                                                         dtype=torch.float32)
    return out


def _isf(c):
    return sf.ISF(_size(c), _dims(c), HBAR, DT)


def _omega_t(omega, k):
    """Float32(omega * Float32(k dt)), as the driver forms it."""
    f = torch.float32
    return float(torch.tensor(omega, dtype=f) * (torch.tensor(float(k), dtype=f) * torch.tensor(DT, dtype=f)))


def _jet(c, k):
    noz = _nozzle(c)
    return {"kvec": noz["kvec"], "omega_t": _omega_t(noz["omega"], k), "cen": noz["cen"], "len": noz["len"],
            "rad": noz["rad"], "phase_mode": sf.PHASE_DOT, "emit_mode": sf.EMIT_DISC}


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = {"case": c, "k": 0, "seed": int(seed), "in": _fields(c, seed)}
    if kind == "batch":
        s["batch"] = sf.ISFBatch(s["in"]["sims"])
        for i in range(c["sims"]):
            s["batch"].set_psi(i, s["in"]["psi"][i])
            s["batch"].set_particles(i, s["in"]["parts"][i])
        return s
    if kind == "matlab":
        s["isf"] = sf.matlabport.ISF(_size(c), _dims(c), HBAR, DT)
        p = s["in"]["psi"].to(torch.float64)
        s["psi"] = tuple(torch.complex(p[..., 2 * i], p[..., 2 * i + 1]).contiguous().permute(2, 1, 0) for i in (0, 1))
        return s
    s["isf"] = _isf(c)
    if kind in ("step", "loop") and c["jet"]:
        s["noz"] = _nozzle(c)
        s["jet"] = _jet(c, 0) | {"emit_count": c["emit"], "seed": int(seed)}
    if kind == "loop":
        s["mask"] = sf.isjet(s["isf"], s["noz"]["cen"], s["noz"]["len"], s["noz"]["rad"])
    if kind == "advect":
        s["noz"] = _nozzle(c)
        s["isf"].velocity = s["in"]["vel"]
    if kind == "adj_step":
        s["jet"] = _jet(c, 3)
    if kind == "adj_gradient":
        noz = _nozzle(c)
        s["problem"] = sf.adj_problem(c["steps"], c["every"], noz["kvec"], noz["omega"],
                                      (noz["cen"], noz["len"], noz["rad"]), init_iters=c["init"])
    return s


# --------------------------------------------------------------------- run
def run(state):
    c, isf, d = state["case"], state.get("isf"), state["in"]
    kind = c["kind"]
    if kind == "flow":
        sf.schroedinger_flow(isf, d["psi"])
        sf.normalize_psi(isf, d["psi"])
        return d["psi"]
    if kind == "project":
        return sf.pressure_project(isf, d["psi"])
    if kind == "velocity":
        sf.velocity_one_form(isf, d["psi"], HBAR)
        sf.staggered_sharp(isf)
        return isf.velocity
    if kind == "step":
        state["k"] += 1
        jet = None
        if c["jet"]:
            k = state["k"]
            jet = state["jet"]
            jet["omega_t"] = state["noz"]["omega"] * (k * DT)
            jet["emit_start"] = ((k - 1) * c["emit"]) % c["slots"]
            jet["counter"] = k
        sf.step(isf, d["psi"], d["parts"], jet)
        return d["psi"], d["parts"]
    if kind == "loop":
        state["k"] += 1
        k, noz, jet = state["k"], state["noz"], state["jet"]
        psi, parts = d["psi"], d["parts"]
        sf.schroedinger_flow(isf, psi)
        sf.normalize_psi(isf, psi)
        sf.pressure_project(isf, psi)
        start = ((k - 1) * c["emit"]) % c["slots"]
        sf.add_particles(isf, parts, range(start, start + c["emit"]), noz["cen"], noz["rad"], seed=state["seed"],
                         counter=k, mode=sf.EMIT_DISC)
        sf.restrict_velocity(isf, psi, noz["kvec"], state["mask"], noz["omega"] * (k * DT), phase_mode=jet["phase_mode"])
        sf.pressure_project(isf, psi)
        sf.velocity_one_form(isf, psi, HBAR)
        sf.staggered_sharp(isf)
        sf.staggered_advect(parts, isf)
        return psi, parts
    if kind == "advect":
        state["k"] += 1
        k, noz = state["k"], state["noz"]
        start = ((k - 1) * c["emit"]) % c["slots"]
        sf.add_particles(isf, d["parts"], range(start, start + c["emit"]), noz["cen"], noz["rad"], seed=state["seed"],
                         counter=k, mode=sf.EMIT_DISC)
        return sf.staggered_advect(d["parts"], isf)
    if kind == "batch":
        b = state["batch"]
        b.step(c["steps"])
        return [(b.psi(i), b.particles(i)) for i in range(c["sims"])]
    if kind == "adj_step":
        psibar, partsbar = d["psibar"].clone(), d["partsbar"].clone()
        jb = sf.adj_step(isf, d["psi"], d["parts"], state["jet"], psibar, partsbar)
        return psibar, partsbar, jb
    if kind == "adj_gradient":
        # the cotangents of kvec and omega are left out: the loss does not depend on them but for round-off
        # (the projection removes every exact one-form), so they hold nothing that can be compared
        loss, gpsi, gparts, _ = sf.adj_gradient(isf, state["problem"], d["psi"], d["parts"], d["targets"])
        return loss, gpsi, gparts
    m = sf.matlabport
    p1, p2 = m.SchroedingerFlow(isf, *state["psi"])
    p1, p2 = m.Normalize(p1, p2)
    p1, p2 = m.PressureProject(isf, p1, p2)
    state["psi"] = (p1, p2)
    v = m.VelocityOneForm(isf, p1, p2, HBAR)
    return p1, p2, m.StaggeredSharp(isf, *v)


# -------------------------------------------------------------------- work
def work(case):
    """psi is 16 B per cell, the velocity 12, a particle 12; FFTs at 5 N log2 N operations per complex field, an angle at 30."""
    c = case
    n = c["nx"] * c["ny"] * c["nz"]
    fft = 5 * n * math.log2(n)
    flow, proj, vel = 4 * fft + 8 * n, fft + 130 * n, 100 * n
    kind, p = c["kind"], c.get("slots", 0)
    if kind == "flow":
        return {"bytes": 32 * n, "flops": flow + 10 * n}
    if kind == "project":
        return {"bytes": 32 * n, "flops": proj}
    if kind == "velocity":
        return {"bytes": 28 * n, "flops": vel}
    if kind in ("step", "loop"):
        # psi and the particles in and out, the velocity out
        return {"bytes": 44 * n + 24 * p, "flops": flow + (2 if c["jet"] else 1) * proj + vel + 250 * p}
    if kind == "advect":
        return {"bytes": 12 * n + 24 * p, "flops": 250 * p}
    if kind == "batch":
        total = {"bytes": 0, "flops": 0}
        for i in range(c["sims"]):
            (nx, ny, nz), _ = cfgs.ENSEMBLE_GRIDS[i % len(cfgs.ENSEMBLE_GRIDS)]
            w = work({"kind": "step", "nx": nx, "ny": ny, "nz": nz, "jet": True, "slots": p})
            total = {k: total[k] + c["steps"] * w[k] for k in total}
        return total
    if kind == "adj_step":
        # psi in, its cotangent in and out; the particles in, their cotangent in and out; twice the step's operations and the reverse sweep
        return {"bytes": 48 * n + 36 * p, "flops": 2 * (2 * flow + 4 * proj + 2 * vel) / 2 + 800 * p}
    if kind == "adj_gradient":
        step = flow + 2 * proj + vel + 250 * p
        return {"bytes": 32 * n + 36 * p, "flops": 3.5 * (c["steps"] * step + c["init"] * proj)}
    # five calls, each with its complex128 / float64 fields in and out
    return {"bytes": (64 + 64 + 64 + 56 + 48) * n, "flops": flow + proj + vel + 10 * n}


# ------------------------------------------------------------------- exact
class _Grid64:
    """The operators in 64 bits (src/parallel.jl, src/particles.jl), plain torch."""

    def __init__(self, c):
        self.dims, self.size = _dims(c), _size(c)
        f32 = lambda v: float(torch.tensor(v, dtype=torch.float32))  # noqa: E731
        self.d = [f32(length / n) for n, length in zip(self.dims, self.size)]
        self.dt = f32(DT)
        ths, s2s = [], []
        for n, length, d in zip(self.dims, self.size, self.d):
            k = torch.arange(n, device=_dev(), dtype=torch.float64)
            ks = torch.where(k < n // 2, k, k - n) / length
            ths.append(-4 * math.pi ** 2 * HBAR * ks * ks * self.dt / 2)
            s2s.append((torch.sin(math.pi * k / n) / d) ** 2)
        add = lambda v: v[0][None, None, :] + v[1][None, :, None] + v[2][:, None, None]  # noqa: E731
        self.mask = torch.polar(torch.ones(self.dims[::-1], device=_dev(), dtype=torch.float64), add(ths))
        den = add(s2s)
        den[0, 0, 0] = 1.0
        self.fac = -0.25 / den
        self.fac[0, 0, 0] = 0.0

    @staticmethod
    def split(psi):
        p = psi.to(torch.float64)
        return torch.complex(p[..., 0], p[..., 1]), torch.complex(p[..., 2], p[..., 3])

    @staticmethod
    def join(p):
        return torch.stack([p[0].real, p[0].imag, p[1].real, p[1].imag], dim=-1)

    def flow(self, p):
        return tuple(torch.fft.ifftn(torch.fft.fftn(q) * self.mask) for q in p)

    @staticmethod
    def normalize(p):
        n = torch.sqrt(p[0].abs() ** 2 + p[1].abs() ** 2)
        return p[0] / n, p[1] / n

    @staticmethod
    def one_form(p, hbar=1.0):
        return [hbar * torch.angle(sum(torch.conj(q) * torch.roll(q, -1, ax) for q in p)) for ax in (2, 1, 0)]

    def project(self, p):
        v = self.one_form(p)
        f = sum((a - torch.roll(a, 1, ax)) / d ** 2 for a, ax, d in zip(v, (2, 1, 0), self.d))
        q = torch.fft.ifftn(torch.fft.fftn(f) * self.fac).real
        g = torch.polar(torch.ones_like(q), -q)
        return p[0] * g, p[1] * g

    def sharp(self, v):
        return [a / d for a, d in zip(v, self.d)]

    def restrict(self, p, noz, kvec, omega_t):
        x, y, z = (torch.arange(n, device=_dev(), dtype=torch.float32) * torch.tensor(d, dtype=torch.float32, device=_dev())
                   for n, d in zip(self.dims, self.d))
        x, y, z = x[None, None, :], y[None, :, None], z[:, None, None]
        cen = [torch.tensor(v, dtype=torch.float32, device=_dev()) for v in noz["cen"]]
        jet = ((x - cen[0]).abs() <= noz["len"] / 2) & ((y - cen[1]) ** 2 + (z - cen[2]) ** 2
                                                       <= torch.tensor(noz["rad"], dtype=torch.float32, device=_dev()) ** 2)
        ph = kvec[0] * x.double() + kvec[1] * y.double() + kvec[2] * z.double() - omega_t
        e = torch.complex(torch.cos(ph), torch.sin(ph))
        return tuple(torch.where(jet, q.abs() * e, q) for q in p)

    def sample(self, pts, vel):
        """staggered_velocity at pts (P, 3); vel (nz, ny, nx, 3)."""
        i, w = [], []
        for a, (n, length, d) in enumerate(zip(self.dims, self.size, self.d)):
            q = torch.remainder(pts[:, a], length)
            k = torch.floor(q.detach() / d).long().clamp(0, n - 1)
            i.append(k)
            w.append(q - k * d)
        j = [(k + 1) % n for k, n in zip(i, self.dims)]
        at = lambda a, x, y, z: vel[z, y, x, a]  # noqa: E731
        (x, y, z), (xp, yp, zp), (wx, wy, wz) = i, j, w
        ux = (1 - wz) * ((1 - wy) * at(0, x, y, z) + wy * at(0, x, yp, z)) + wz * ((1 - wy) * at(0, x, y, zp) + wy * at(0, x, yp, zp))
        uy = (1 - wz) * ((1 - wx) * at(1, x, y, z) + wx * at(1, xp, y, z)) + wz * ((1 - wx) * at(1, x, y, zp) + wx * at(1, xp, y, zp))
        uz = (1 - wy) * ((1 - wx) * at(2, x, y, z) + wx * at(2, xp, y, z)) + wy * ((1 - wx) * at(2, x, yp, z) + wx * at(2, xp, yp, z))
        return torch.stack([ux, uy, uz], 1)

    def advect(self, p, vel):
        box = torch.tensor(self.size, device=_dev(), dtype=torch.float64)
        inside = ((p > 0) & (p < box)).all(1, keepdim=True)
        k1 = self.sample(p, vel)
        k2 = self.sample(p + k1 * self.dt * 0.5, vel)
        k3 = self.sample(p + k2 * self.dt * 0.5, vel)
        k4 = self.sample(p + k3 * self.dt, vel)
        return torch.where(inside, p + self.dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4), -1.0)


def _step64(e, p, noz, kvec, omega_t):
    p = e.project(e.normalize(e.flow(p)))
    return p if noz is None else e.project(e.restrict(p, noz, kvec, omega_t))


def exact(case, seed):
    """Positions of particles have no 64-bit counterpart in the cases that carry them through a computed velocity: the
    reference's interpolation jumps at cell faces, so one rounding away a particle goes another way.  Where the
    velocity is given (the advection on its own) the births are the library's own random stream."""
    c, kind = case, case["kind"]
    if kind == "advect":
        return None
    d = _fields(c, seed)
    if kind == "batch":
        out = []
        for i, s in enumerate(d["sims"]):
            ci = dict(zip(("nx", "ny", "nz", "lx", "ly", "lz"), tuple(s["dims"]) + tuple(s["physical_size"])))
            e, p = _Grid64(ci), _Grid64.split(d["psi"][i])
            for k in range(1, c["steps"] + 1):
                p = _step64(e, p, s["jet"], s["jet"]["kvec"], _omega_t(s["jet"]["omega"], k))
            out.append((e.join(p), None))
        return out
    e = _Grid64(c)
    p = e.split(d["psi"])
    if kind == "flow":
        return e.join(e.normalize(e.flow(p)))
    if kind == "project":
        return e.join(e.project(p))
    if kind == "velocity":
        return torch.stack(e.sharp(e.one_form(p, HBAR)), dim=-1)
    if kind in ("step", "loop"):
        noz = _nozzle(c) if c["jet"] else None
        w = None if noz is None else float(torch.tensor(noz["omega"] * DT, dtype=torch.float32))
        return e.join(_step64(e, p, noz, noz and noz["kvec"], w)), None
    if kind == "matlab":
        p = e.project(e.normalize(e.flow(p)))
        v = e.sharp(e.one_form(p, HBAR))
        return p[0].permute(2, 1, 0), p[1].permute(2, 1, 0), tuple(a.permute(2, 1, 0) for a in v)
    noz = _nozzle(c)
    if kind == "adj_step":
        psi = d["psi"].to(torch.float64).requires_grad_()
        parts = d["parts"].to(torch.float64).requires_grad_()
        jp = torch.tensor(noz["kvec"] + (_omega_t(noz["omega"], 3),), device=_dev(), dtype=torch.float64, requires_grad=True)
        p = _step64(e, e.split(psi), noz, jp[:3], jp[3])
        out = e.advect(parts, torch.stack(e.sharp(e.one_form(p, HBAR)), dim=-1))
        total = (e.join(p) * d["psibar"].double()).sum() + (out * d["partsbar"].double()).sum()
        g = torch.autograd.grad(total, (psi, parts, jp))
        return g[0], g[1], g[2].tolist()
    psi = d["psi"].to(torch.float64).requires_grad_()
    parts0 = d["parts"].to(torch.float64).requires_grad_()
    p, parts = e.split(psi), parts0
    for _ in range(c["init"]):
        p = e.project(e.restrict(p, noz, noz["kvec"], 0.0))
    for k in range(1, c["steps"] + 1):
        p = _step64(e, p, noz, noz["kvec"], _omega_t(noz["omega"], k))
        parts = e.advect(parts, torch.stack(e.sharp(e.one_form(p, HBAR)), dim=-1))
    alive = (parts[:, :1] >= 0).detach()
    loss = (torch.where(alive, parts - d["targets"].double(), 0.0) ** 2).sum()
    g = torch.autograd.grad(loss, (psi, parts0))
    return float(loss.detach()), g[0], g[1]
