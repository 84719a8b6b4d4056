"""What a user of the solver has it do, as measurable cases.

A case is one pass through public entry points: particles are handed over, the
solver advances some frames, positions and velocities are read back (or, for
the differentiable rollout, gradients; for the grid build, the sorted order
and the cell table).  Sizes run from a thousand particles, where a step is
bound by latency and launches, to eight million.  Scenes are dam breaks with
the repository's parameters (h = 0.1, lattice spacing 0.5 h), its scaled
variants, the reference's benchmark scene, the imbalanced blob scene and the
batch of uneven scenes.

``warm`` frames are run once while a case is prepared, so that the measured
frames start from a flow in motion (disordered, compressed at the walls); with
``warm`` 0 the particles are a jittered lattice in a swirling motion, made from
the seed alone, for which ``exact`` computes the step in 64 bits.
"""

from __future__ import annotations

import ctypes
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
H = 0.1
SPACING = 0.5 * H
RADIUS = 0.025


def _package():
    """The package directory has a hyphen in its name, so it is loaded by path."""
    name = "fluid_simulator_gb300"
    if name not in sys.modules:
        path = os.path.join(ROOT, "fluid-simulator_gb300")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(path, "__init__.py"), submodule_search_locations=[path])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _module(name):
    _package()
    return importlib.import_module("fluid_simulator_gb300." + name)


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def _dam(name, nx, ny, nz, **kw):
    case = dict(name=name, kind="dam", nx=nx, ny=ny, nz=nz, frames=1, warm=0, iterations=4,
                substeps=1, xsph=True, vorticity=True, scorr_n=4, colliders=False, host=False)
    case.update(kw)
    return case


def listed():
    return [
        # One step of the smallest scenes (the size of the repository's
        # stability scenario and of its smoke test): latency and launches.
        _dam("step_1k", 16, 8, 8),
        # A ragged scene between the tuned sizes, three iterations, no vorticity.
        _dam("step_11k_odd", 29, 23, 17, iterations=3, vorticity=False),
        # The 16,384-particle dam break in motion, several frames per call.
        _dam("run_16k", 32, 32, 16, frames=10, warm=60),
        # A mid-size scene, one frame per call as an interactive program steps it.
        _dam("step_65k", 64, 64, 16, warm=60),
        # The reference's own benchmark scene: 262,144 particles, two
        # substeps, a box and a sphere.
        dict(name="reference_262k", kind="reference", layers=32, frames=2, warm=30),
        # The headline workload: 1,048,576 particles in motion.
        _dam("run_1m", 128, 128, 64, frames=4, warm=60),
        # The same scene driven with host buffers: upload, one step, download.
        _dam("host_1m", 128, 128, 64, warm=60, host=True),
        # Strongly uneven cell occupancy at 8.4 M particles, compact lists,
        # once the blobs' first burst is over.
        dict(name="imbalanced_8m", kind="imbalanced", n=8_388_608, blobs=16, frames=1, warm=10,
             lists="compact"),
        # Hundreds of scenes of uneven size stepped together.
        dict(name="batch_256", kind="batch", scenes=256, n_min=2048, n_max=65536, frames=2),
        # Differentiable rollout, the gradient of a small scene: forward and
        # backward with a checkpoint every two steps.
        dict(name="grad_4k", kind="grad", nx=15, ny=16, nz=17, steps=4, every=2, vorticity=True,
             colliders=False),
        # The 65,536-particle rollout with checkpoints every ten steps.
        dict(name="grad_65k", kind="grad", nx=64, ny=64, nz=16, steps=20, every=10,
             vorticity=True, colliders=False),
        # The grid build alone on device arrays: cell keys, stable sort, cell table.
        dict(name="grid_200k", kind="grid", n=200_003, gx=96, gy=48, gz=40),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, lo, hi):
    """Lattice dimensions of a block of about log-uniform size, odd ones among them."""
    n = _log(rng, lo, hi)
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    side = n ** (1.0 / 3.0)
    nx, ny = max(4, round(side * a)), max(4, round(side * b))
    return nx, ny, max(4, round(n / (nx * ny)))


def draw(rng):
    kind = rng.choices(["dam", "host", "reference", "imbalanced", "batch", "grad", "grid"],
                       [8, 2, 1, 2, 2, 3, 2])[0]
    if kind in ("dam", "host"):
        nx, ny, nz = _block(rng, 1000, 1_000_000)
        large = nx * ny * nz > 200_000
        case = _dam("", nx, ny, nz, frames=rng.choice([1, 2, 3] if large else [1, 2, 5, 8]),
                    warm=rng.choice([0, 20, 60]), iterations=rng.choice([2, 3, 4, 4, 5]),
                    substeps=1 if large else rng.choice([1, 1, 2]),
                    xsph=rng.random() < 0.8, vorticity=rng.random() < 0.8,
                    scorr_n=rng.choice([0, 2, 4, 4, 5]), colliders=rng.random() < 0.4,
                    host=kind == "host")
        if case["host"]:
            case["frames"] = 1
        del case["name"]
        return case
    if kind == "reference":
        return dict(kind=kind, layers=rng.randint(4, 32), frames=rng.choice([1, 2]),
                    warm=rng.choice([10, 30]))
    if kind == "imbalanced":
        n = int(_log(rng, 100_000, 1_500_000))
        lists = rng.choice(["compact", "slots"]) if n < 1_000_000 else "compact"
        return dict(kind=kind, n=n, blobs=max(2, n // 500_000), frames=1,
                    warm=rng.choice([0, 2, 10]), lists=lists)
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(8, 200), n_min=rng.choice([500, 1000, 2048]),
                    n_max=rng.choice([8192, 20000, 65536]), frames=rng.choice([1, 2]))
    if kind == "grad":
        nx, ny, nz = _block(rng, 800, 40_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randint(2, 12),
                    every=rng.randint(2, 6), vorticity=rng.random() < 0.7,
                    colliders=rng.random() < 0.3)
    return dict(kind=kind, n=int(_log(rng, 500, 262_144)), gx=rng.randint(8, 120),
                gy=rng.randint(8, 80), gz=rng.randint(8, 80))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _params(case):
    """The repository's dam-break parameters with the case's options."""
    P = _module("scenes").dam_break_params()
    P.solverIterations = case.get("iterations", 4)
    P.substeps = case.get("substeps", 1)
    if not case.get("xsph", True):
        P.xsphViscosity = 0.0
    if not case.get("vorticity", True):
        P.vorticityStrength = 0.0
    n = case.get("scorr_n", 4)
    if n:
        P.scorrN = n
    else:
        P.scorrK, P.scorrN, P.scorrDeltaQ = 0.0, 0, 0.0
    return P


def _lattice(nx, ny, nz, jitter, rng):
    z, y, x = np.meshgrid(np.arange(nz, dtype=np.float32), np.arange(ny, dtype=np.float32),
                          np.arange(nx, dtype=np.float32), indexing="ij")
    pos = np.ones((nx * ny * nz, 4), np.float32)
    for a, c in enumerate((x, y, z)):
        pos[:, a] = c.ravel() * np.float32(SPACING) + np.float32(RADIUS)
    pos[:, :3] += (rng.random((pos.shape[0], 3), np.float32) * 2 - 1) * np.float32(jitter)
    return pos


def _swirl(pos, rng, speed):
    """A smooth velocity field with shear and vorticity, random in phase."""
    vel = np.zeros_like(pos)
    k = rng.uniform(1.0, 3.0, (3, 2))
    ph = rng.uniform(0.0, 2.0 * np.pi, (3, 2))
    for a in range(3):
        u, w = pos[:, (a + 1) % 3].astype(np.float64), pos[:, (a + 2) % 3].astype(np.float64)
        vel[:, a] = speed * (np.sin(k[a, 0] * u + ph[a, 0]) + np.cos(k[a, 1] * w + ph[a, 1]))
    return vel


def _dam_inputs(case, seed):
    """(positions, velocities, low, high): a block in a box twice as wide and deep."""
    rng = np.random.default_rng([seed, 11])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    still = case.get("warm", 0) > 0
    pos = _lattice(nx, ny, nz, 0.01 * H if still else 0.12 * SPACING, rng)
    vel = np.zeros_like(pos) if still else _swirl(pos, rng, 0.4)
    return pos, vel, (0.0, 0.0, 0.0), (2 * nx * SPACING, ny * SPACING, 2 * nz * SPACING)


def _dam_colliders(hi):
    """A sphere in the block's path, a box on the floor and a tilted plane."""
    r = 0.15 * min(hi)
    return dict(spheres=[((0.7 * hi[0], 0.5 * r, 0.4 * hi[2]), r)],
                boxes=[((0.75 * hi[0], 0.1 * hi[1], 0.8 * hi[2]),
                        (0.05 * hi[0], 0.1 * hi[1], 0.05 * hi[2]))],
                planes=[((0.95 * hi[0], 0.0, 0.5 * hi[2]), (-0.8, 0.6, 0.0))])


def _imbalanced_inputs(case, seed):
    """Half a dense lattice column, half Gaussian blobs of sigma 4 h (about
    1,090 neighbours at a blob's centre), each blob in its own part of the box."""
    rng = np.random.default_rng([seed, 12])
    half = case["n"] // 2
    side = max(8, round((half / 2) ** (1.0 / 3.0)))
    col = _lattice(side, max(1, half // (side * side)), side, 0.01 * H, rng)
    rest, blobs = case["n"] - col.shape[0], case["blobs"]
    # A blob of sigma s holds (s / 4 h)^3 of the 262,144 particles of the full one.
    sigma = 4 * H * (rest / blobs / 262_144.0) ** (1.0 / 3.0)
    part = 16.0 * sigma
    gx = max(1, math.ceil((2 * blobs) ** (1.0 / 3.0)))
    gz = max(1, math.ceil(math.sqrt(blobs / gx)))
    gy = max(1, math.ceil(blobs / (gx * gz)))
    hi = (max(gx * part, 2 * side * SPACING), max(gy * part, 1.05 * col[:, 1].max()),
          max(gz * part, 1.5 * side * SPACING))
    at = np.arange(blobs)
    cell = np.stack([at % gx, at // (gx * gz), at // gx % gz], 1).astype(np.float64)
    centre = (cell + 0.5 + rng.uniform(-0.2, 0.2, (blobs, 3))) * part
    pos = np.ones((case["n"], 4), np.float32)
    pos[:col.shape[0]] = col
    which = rng.integers(0, blobs, rest)
    blob = centre[which].astype(np.float32)
    blob += rng.standard_normal((rest, 3), np.float32) * np.float32(sigma)
    pos[col.shape[0]:, :3] = np.clip(blob, RADIUS, np.asarray(hi, np.float32) - RADIUS)
    return pos, np.zeros_like(pos), (0.0, 0.0, 0.0), tuple(float(v) for v in hi)


def _batch_inputs(case, seed):
    pkg, common = _package(), _module("scenes").dam_break_params()
    # The sizes are the case's; the seed moves the particles and the densities.
    sizes = np.exp(np.random.default_rng([case["scenes"], case["n_min"], case["n_max"]]).uniform(
        np.log(case["n_min"]), np.log(case["n_max"]), case["scenes"]))
    rng = np.random.default_rng([seed, 13])
    scenes, pos, vel = [], [], []
    for n in sizes:
        k = max(2, int(round((n / 4.0) ** (1.0 / 3.0))))
        p = _lattice(2 * k, 2 * k, k, 0.08 * SPACING, rng)
        rho = float(np.float32(common.restDensity * rng.uniform(0.9, 1.1)))
        mass = float(np.float32(rho) * np.float32(SPACING) ** 3)
        xsph = float(np.float32(rng.uniform(0.005, 0.05) * mass / rho))
        scenes.append(pkg.Scene(len(p), (0.0, 0.0, 0.0),
                                (4 * k * SPACING, 2 * k * SPACING, 2 * k * SPACING), rho, mass,
                                xsph))
        pos.append(p)
        vel.append(_swirl(p, rng, 0.3))
    return scenes, common, np.concatenate(pos), np.concatenate(vel)


def _grad_inputs(case, seed):
    """Initial state and the gradient of a mean squared distance at the end."""
    pos, vel, lo, hi = _dam_inputs(case, seed)
    rng = np.random.default_rng([seed, 14])
    gx, gv = np.zeros_like(pos), np.zeros_like(pos)
    gx[:, :3] = (2.0 / len(pos)) * (rng.standard_normal((len(pos), 3)) * 0.05 - (0.3, 0.0, 0.0))
    gv[:, :3] = (1e-3 / len(pos)) * rng.standard_normal((len(pos), 3))
    return pos, vel, lo, hi, gx, gv


def _grid_inputs(case, seed):
    rng = np.random.default_rng([seed, 15])
    cell = 0.1
    hi = (case["gx"] * cell * 0.999, case["gy"] * cell * 0.999, case["gz"] * cell * 0.999)
    pos = np.ones((case["n"], 4), np.float32)
    pos[:, :3] = rng.uniform((-0.05,) * 3, np.asarray(hi) + 0.05, (case["n"], 3))
    return pos, (0.0, 0.0, 0.0), hi, cell


# ---------------------------------------------------------------------------
# Preparing and running
# ---------------------------------------------------------------------------

def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float32, pin_memory=True)
    t.numpy()[...] = a
    return t


def _device(a):
    return torch.from_numpy(a).cuda()


def prepare(case, seed):
    pkg, kind = _package(), case["kind"]
    if kind == "grid":
        pos, lo, hi, cell = _grid_inputs(case, seed)
        dims = pkg.grid_dims(lo, hi, cell)
        out = [torch.empty(case["n"], dtype=torch.int32, device="cuda") for _ in range(2)]
        out += [torch.empty(math.prod(dims), dtype=torch.int32, device="cuda") for _ in range(2)]
        return dict(kind=kind, x=_device(pos), lo=pkg.Float3(*lo), hi=pkg.Float3(*hi), cell=cell,
                    out=out, lib=pkg.load())
    if kind == "grad":
        pos, vel, lo, hi, gx, gv = _grad_inputs(case, seed)
        prm = _params(case)
        a = pkg.PBFAdjoint()
        a.initialize(len(pos), lo, hi, prm, max_neighbors=128, checkpoint_every=case["every"])
        if case["colliders"]:
            c = _dam_colliders(hi)
            a.set_spheres(c["spheres"])
            a.set_boxes(c["boxes"])
            a.set_planes(c["planes"])
        ins = [_device(pos), _device(vel), torch.tensor(prm.restDensity, dtype=torch.float64),
               torch.tensor(prm.xsphViscosity, dtype=torch.float64)]
        for t in ins:
            t.requires_grad_()
        return dict(kind=kind, adjoint=a, ins=ins, steps=case["steps"],
                    seeds=[_device(gx), _device(gv)], rollout=_module("autograd").rollout)

    s = pkg.PBFSolver()
    if kind == "dam":
        pos, vel, lo, hi = _dam_inputs(case, seed)
        s.initialize(len(pos), lo, hi, _params(case))
        if case["colliders"]:
            c = _dam_colliders(hi)
            s.set_spheres(c["spheres"])
            s.set_boxes(c["boxes"])
            s.set_planes(c["planes"])
    elif kind == "reference":
        # The scene has no random part: a small jitter makes the seeds differ.
        pos, vel, lo, hi, prm, c = _module("scenes").reference_benchmark(case["layers"] * 8192)
        rng = np.random.default_rng([seed, 16])
        pos[:, :3] += rng.uniform(-1e-3, 1e-3, (len(pos), 3)).astype(np.float32)
        s.initialize(len(pos), lo, hi, prm)
        s.set_boxes(c["boxes"])
        s.set_spheres(c["spheres"])
    elif kind == "imbalanced":
        pos, vel, lo, hi = _imbalanced_inputs(case, seed)
        cap = min(400 * len(pos), 2 ** 32 - 1) if case["lists"] == "compact" else None
        s.initialize(len(pos), lo, hi, _module("scenes").dam_break_params(), max_neighbors=2048,
                     list_capacity=cap)
    else:
        scenes, common, pos, vel = _batch_inputs(case, seed)
        s.initialize_batch(scenes, common)
    state = dict(kind="step", solver=s, frames=case["frames"], host=case.get("host", False))
    warm = case.get("warm", 0)
    if warm:
        s.set_particles(pos, vel)
        s.run(warm)
        pos, vel = s.copy_positions_to_host(), s.copy_velocities_to_host()
    if state["host"]:
        state["keep"] = [_pinned(pos), _pinned(vel), _pinned(pos), _pinned(vel)]
        state["x"], state["v"], state["xo"], state["vo"] = (t.numpy() for t in state["keep"])
    else:
        state["x"], state["v"] = _device(pos), _device(vel)
        state["xo"], state["vo"] = torch.empty_like(state["x"]), torch.empty_like(state["v"])
    return state


def run(state):
    if state["kind"] == "grid":
        a = [ctypes.c_void_p(t.data_ptr()) for t in state["out"]]
        st = state["lib"].pbf_grid_build_static_scratch(
            ctypes.c_void_p(state["x"].data_ptr()), state["x"].shape[0], state["lo"], state["hi"],
            state["cell"], *a, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st:
            raise RuntimeError("the grid build returned %d" % st)
        return state["out"]
    if state["kind"] == "grad":
        x, v = state["rollout"](state["adjoint"], *state["ins"], state["steps"])
        grads = torch.autograd.grad([x, v], state["ins"], state["seeds"])
        return [x.detach(), v.detach(), *grads]
    s = state["solver"]
    if state["host"]:
        s.set_particles(state["x"], state["v"])
        s.run(state["frames"])
        s.copy_positions_to_host(out=state["xo"])
        s.copy_velocities_to_host(out=state["vo"])
    else:
        s.set_particles_device(state["x"], state["v"])
        s.run(state["frames"])
        s.copy_positions_device(state["xo"])
        s.copy_velocities_device(state["vo"])
    return [state["xo"], state["vo"]]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

NEIGHBOURS = 33  # within h at the rest spacing of 0.5 h


def _step_flops(n, iterations, xsph, vorticity, neighbours=NEIGHBOURS):
    """Pair arithmetic of a substep: per iteration the distance (8), density
    and gradient sums (25) and the position correction (30); at the end the
    distance again, XSPH (13), vorticity (35) and confinement (30)."""
    post = (8 if xsph or vorticity else 0) + (13 if xsph else 0) + (65 if vorticity else 0)
    return n * neighbours * (iterations * 63.0 + post)


def work(case):
    kind, frames = case["kind"], case.get("frames", 1)
    if kind == "grid":
        cells = case["gx"] * case["gy"] * case["gz"]
        return dict(bytes=24.0 * case["n"] + 8.0 * cells, flops=6.0 * case["n"])
    if kind == "grad":
        # Forward and reverse: the state in, the state out and the gradients
        # of each step; the reverse pass costs about twice the pair arithmetic.
        n, steps = case["nx"] * case["ny"] * case["nz"], case["steps"]
        return dict(bytes=128.0 * n * steps,
                    flops=3.0 * steps * _step_flops(n, 4, True, case["vorticity"]))
    if kind == "dam":
        n, subs = case["nx"] * case["ny"] * case["nz"], case["substeps"]
        flops = _step_flops(n, case["iterations"], case["xsph"], case["vorticity"])
    elif kind == "reference":
        n, subs = case["layers"] * 8192, 2
        flops = _step_flops(n, 4, True, True)
    elif kind == "imbalanced":
        n, subs = case["n"], 1
        flops = _step_flops(n, 4, True, True, 0.5 * (NEIGHBOURS + 400))
    else:
        lo, hi = case["n_min"], case["n_max"]
        n, subs = case["scenes"] * (hi - lo) / math.log(hi / lo), 1
        flops = _step_flops(n, 4, True, True)
    # A substep reads the state (32 bytes a particle) and writes it.
    return dict(bytes=64.0 * n * frames * subs, flops=flops * frames * subs)


# ---------------------------------------------------------------------------
# The step in 64 bits
# ---------------------------------------------------------------------------

def _pairs(x, h2):
    """Indices (i, j) of all pairs i != j closer than h."""
    found = []
    n = x.shape[0]
    for a in range(0, n, 1024):
        d2 = ((x[a:a + 1024, None, :] - x[None, :, :]) ** 2).sum(2)
        i, j = torch.nonzero(d2 <= h2, as_tuple=True)
        i = i + a
        keep = i != j
        found.append((i[keep], j[keep]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _exact_step(x, v, q, lo, hi, rho0, xsph):
    """One substep of the solver's formulas; q: the other parameters as doubles."""
    h, dt = q["h"], q["dt"]
    h2 = h * h
    c6, cs = 315.0 / (64.0 * math.pi * h ** 3), -45.0 / (math.pi * h ** 4)
    n = x.shape[0]
    gs = q["mass"] / rho0

    def total(i, term):
        return torch.zeros((n,) + tuple(term.shape[1:]), dtype=x.dtype,
                           device=x.device).index_add(0, i, term)

    def geometry(p):
        with torch.no_grad():
            i, j = _pairs(p, h2)
        r = p[i] - p[j]
        d2 = (r * r).sum(1)
        w = c6 * (1.0 - d2 / h2) ** 3
        rr = torch.sqrt(d2)
        g = (cs * (1.0 - rr / h) ** 2 / rr)[:, None] * r
        return i, j, d2, w, g

    low, high = q["low"], q["high"]  # the container less the particle radius
    v1 = v + q["gravity"] * dt
    p = x + v1 * dt
    for _ in range(q["iterations"]):
        i, j, d2, w, g = geometry(p)
        rho = q["mass"] * (c6 + total(i, w))
        S = total(i, (g * g).sum(1)) + (total(i, g) ** 2).sum(1)
        lam = -(rho / rho0 - 1.0) / (gs * gs * S + q["eps"])
        coef = lam[i] + lam[j]
        if q["k"]:
            coef = coef - q["k"] * ((h2 - d2) / (h2 - q["dq"] ** 2)) ** (3 * q["n"])
        p = p + gs * total(i, coef[:, None] * g)
        p = torch.minimum(torch.maximum(p, low), high)
    u = (p - x) / dt
    i, j, d2, w, g = geometry(p)
    if q["has_xsph"]:
        u = u + xsph * total(i, (u[j] - u[i]) * w[:, None])
    if q["vort"]:
        om = total(i, torch.linalg.cross(g, u[j] - u[i]))
        size = torch.sqrt((om * om).sum(1) + 1e-300)
        eta = total(i, (size[j] - size[i])[:, None] * g)
        length = torch.sqrt((eta * eta).sum(1) + 1e-300)
        unit = torch.where((length > 1e-6)[:, None], eta / length[:, None], torch.zeros_like(eta))
        u = u + dt * q["vort"] * torch.linalg.cross(unit, om)
    # Contacts with the walls: the normal velocity is taken out (restitution
    # 0), the tangential one loses its share to friction.  The top is open.
    for a in range(3):
        for side in (1.0, -1.0):
            if a == 1 and side < 0:
                continue
            near = (p[:, a] <= low[a] + 1e-4) if side > 0 else (p[:, a] >= high[a] - 1e-4)
            vn, vin = u[:, a] * side, v1[:, a] * side
            act = near & ((vn < 0) | ((vn == 0) & (vin < 0)))
            keep = torch.ones(3, dtype=x.dtype, device=x.device)
            keep[a] = 0.0
            u = torch.where(act[:, None], u * keep * (1.0 - q["friction"]), u)
    return p, u


def _exact_parameters(case, prm, lo, hi, device):
    f = lambda v: float(np.float32(v))  # noqa: E731 -- parameters are 32-bit values
    r = np.float32(prm.particleRadius)
    low = np.asarray(lo, np.float32) + r
    high = np.asarray(hi, np.float32) - r
    high[1] = np.inf
    t = lambda a: torch.tensor(np.asarray(a, np.float64), device=device)  # noqa: E731
    return dict(h=f(prm.smoothingRadius), dt=f(np.float32(prm.dt) / np.float32(prm.substeps)),
                mass=f(prm.particleMass), eps=f(prm.lambdaEpsilon), k=f(prm.scorrK), n=prm.scorrN,
                dq=f(prm.scorrDeltaQ), vort=f(prm.vorticityStrength),
                friction=f(np.float32(1) - (np.float32(1) - np.float32(prm.collisionFriction))),
                has_xsph=prm.xsphViscosity != 0.0, iterations=prm.solverIterations,
                gravity=t(np.asarray(prm.gravity, np.float32)), low=t(low), high=t(high))


def exact(case, seed):
    kind = case["kind"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind not in ("dam", "grad") or case["colliders"]:
        return None
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "dam" and (case["warm"] or case["frames"] * case["substeps"] > 2 or n > 40_000):
        return None
    if kind == "grad" and (n > 6000 or case["steps"] > 6):
        return None
    prm = _params(case)
    if kind == "dam":
        pos, vel, lo, hi = _dam_inputs(case, seed)
    else:
        pos, vel, lo, hi, gx, gv = _grad_inputs(case, seed)
    q = _exact_parameters(case, prm, lo, hi, device)
    f64 = lambda a: torch.tensor(a[:, :3].astype(np.float64), device=device)  # noqa: E731
    x0, v0 = f64(pos), f64(vel)
    rho0 = torch.tensor(float(np.float32(prm.restDensity)), dtype=torch.float64, device=device)
    xsph = torch.tensor(float(np.float32(prm.xsphViscosity)), dtype=torch.float64, device=device)
    ins = [x0, v0, rho0, xsph]
    with torch.set_grad_enabled(kind == "grad"):
        if kind == "grad":
            for t in ins:
                t.requires_grad_()
        x, v = x0, v0
        for _ in range(case["steps"] if kind == "grad" else case["frames"] * case["substeps"]):
            x, v = _exact_step(x, v, q, lo, hi, rho0, xsph)

    def four(a, w):
        """(n, 3) with the payload column that the solver returns beside it."""
        return torch.cat([a.detach(), torch.full((n, 1), w, dtype=a.dtype, device=a.device)], 1)

    if kind == "dam":
        return [four(x, 1.0), four(v, 0.0)]
    g = torch.autograd.grad([x, v], ins, [f64(gx), f64(gv)])
    return [four(x, 1.0), four(v, 0.0), four(g[0], 0.0), four(g[1], 0.0), g[2].cpu(), g[3].cpu()]
