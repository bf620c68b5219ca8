"""Performance cases of the PIC step library: what its users have it do.

Each case is one pass through the public entry points (include/picgb.h,
picgb.py), as a caller's program makes it:

  deposit  pgb_deposit_static: the charge grid of particle records that are
           already on the device (a viewer or diagnostic hook between steps)
  fields   a given charge density to potential and field: pgb_set_rho,
           pgb_poisson, pgb_efield and the three grids read back
  phases   one iteration driven call by call, as a host driver written
           against the reference's classes makes it (pic.cpp:1069-1250)
  run      a restart: both species loaded from the records of a dump, the
           pre-loop boundary pass, N steps, and the dump and the grids at
           the end (pic::pic with restart, pic_run, dump_data)
  batch    the same for several independent runs stepped together
           (pgb_step_batch)
  frame    the viewer's plots of a running simulation (pgb_render)

The plasmas are those of bench.py and of the reference's parameters.h: argon
in absorbing walls, hydrogen with the collisional boundary, and the default
preset (collisionless argon with steady-state walls).  Grids are 2^k + 1
nodes a side, as the reference requires; particle counts are what is odd and
ragged.  The macro-particle size always gives the design density 1e15 m^-3.
Records and grids cross the boundary in pinned host buffers that the caller
keeps.
"""
import ctypes
import math
import os
import random
import sys

# many runs on their own streams: 32 hardware work queues (read when the CUDA
# context is created), as bench.py sets them
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import torch

_REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_REPO, "vectorized-particle-in-cell-code-with-graphics_gb300"))
import picgb  # noqa: E402

_EPS0 = 8.854e-12
_GRIDS = ("q_e", "q_i", "rho", "phi", "ex", "ey")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: a hook between steps of a small run
        {"name": "deposit_65", "kind": "deposit", "nodes": 65, "particles": 20000, "order": "random"},
        # the same hook on a large run whose records came from a sorted dump
        {"name": "deposit_513", "kind": "deposit", "nodes": 513, "particles": 6000011, "order": "binned"},
        # a field solve in the reference's own arithmetic on a small grid
        {"name": "fields_65_ref", "kind": "fields", "nodes": 65, "poisson": "FMG_REF", "passes": 1, "walls": 0.0},
        # the converged multigrid mode with driven walls on the large grid
        {"name": "fields_513_dc", "kind": "fields", "nodes": 513, "poisson": "FP32_DC", "passes": 4, "walls": 10.0},
        # a host driver that makes every reference call itself
        {"name": "phases_129", "kind": "phases", "nodes": 129, "particles": 300007, "poisson": "DST_DC", "passes": 2,
         "magnetic": 0.0},
        # bench.py's small configuration: latency and launches count
        {"name": "run_ar_65", "kind": "run", "plasma": "argon", "nodes": 65, "particles": 200000,
         "poisson": "FMG_REF", "passes": 1, "sort": 12, "dti": 1.0, "magnetic": 0.0, "steps": 200},
        # the reference's default preset with its magnetic field on, default
        # run controls (no sort), ragged count
        {"name": "run_default_257", "kind": "run", "plasma": "default", "nodes": 257, "particles": 301003,
         "poisson": "FMG_REF", "passes": 1, "sort": 0, "dti": 1.0, "magnetic": 0.01, "steps": 100},
        # hydrogen with the collisional boundary, ions every other step
        {"name": "run_h_129", "kind": "run", "plasma": "hydrogen", "nodes": 129, "particles": 777777,
         "poisson": "FP32_DC", "passes": 5, "sort": 8, "dti": 2.0, "magnetic": 0.0, "steps": 100},
        # bench.py's mid configuration
        {"name": "run_ar_257", "kind": "run", "plasma": "argon", "nodes": 257, "particles": 4194304,
         "poisson": "DST_DC", "passes": 2, "sort": 12, "dti": 1.0, "magnetic": 0.0, "steps": 100},
        # bench.py's headline configuration
        {"name": "run_h_513", "kind": "run", "plasma": "hydrogen", "nodes": 513, "particles": 16777216,
         "poisson": "DST_DC", "passes": 2, "sort": 12, "dti": 1.0, "magnetic": 0.0, "steps": 96},
        # a parameter study: independent argon runs stepped together
        {"name": "batch_8", "kind": "batch", "runs": 8, "mix": 1004, "most": 1000000, "poisson": "DST_DC",
         "passes": 2, "sort": 8, "steps": 50},
        # three viewer plots of a mid-size run
        {"name": "frame_257", "kind": "frame", "nodes": 257, "particles": 1500003, "pixels": 768, "points": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _solver(rng):
    mode = rng.choice(["FMG_REF", "FMG32", "FP32_DC", "DST_DC", "DST_DC"])
    return mode, {"FMG_REF": 1, "FMG32": 1, "FP32_DC": rng.choice([4, 5]), "DST_DC": rng.choice([1, 2, 2, 3])}[mode]


def draw(rng):
    kind = rng.choice(["deposit", "fields", "phases", "run", "run", "run", "batch", "frame"])
    nodes = rng.choice([65, 129, 257, 513])
    if kind == "deposit":
        return {"kind": kind, "nodes": rng.choice([17, 33, nodes, nodes]), "particles": _log_int(rng, 1000, 8000000),
                "order": rng.choice(["random", "binned"])}
    mode, passes = _solver(rng)
    if kind == "fields":
        return {"kind": kind, "nodes": nodes, "poisson": mode, "passes": passes,
                "walls": round(rng.choice([0.0, rng.uniform(0.1, 50.0)]), 3)}
    if kind == "phases":
        return {"kind": kind, "nodes": nodes, "particles": _log_int(rng, 20000, 2000000), "poisson": mode,
                "passes": passes, "magnetic": rng.choice([0.0, 0.0, 0.02])}
    if kind == "run":
        n = _log_int(rng, 50000, 8000000)
        # at least three particles a cell, and a bounded number of particle-steps
        nodes = max(k for k in (65, 129, 257, 513) if k == 65 or (k <= nodes and n >= 3 * k * k))
        return {"kind": kind, "plasma": rng.choice(["argon", "hydrogen", "default"]), "nodes": nodes, "particles": n,
                "poisson": mode, "passes": passes, "sort": rng.choice([0, 8, 12]), "dti": rng.choice([1.0, 1.0, 2.0]),
                "magnetic": rng.choice([0.0, 0.0, 0.01]), "steps": min(50 if nodes == 513 else 100, max(25, int(2.5e8 / n)))}
    if kind == "batch":
        return {"kind": kind, "runs": rng.randint(3, 10), "mix": rng.randrange(1 << 20),
                "most": _log_int(rng, 100000, 1500000), "poisson": mode, "passes": passes,
                "sort": rng.choice([0, 8, 12]), "steps": rng.randint(20, 40)}
    return {"kind": "frame", "nodes": nodes, "particles": _log_int(rng, 50000, 4000000),
            "pixels": rng.randint(300, 1200), "points": rng.choice([0, 5000])}


# ------------------------------------------------------------ parameters, states
def _params(case, seed, nodes=None, particles=None, torr=0.01, te=2.0):
    nodes, n = nodes or case["nodes"], particles or case["particles"]
    kw = dict(X_NO_OF_CELLS=nodes, RAND_SEED=1 + seed % 100003, POISSON=case["poisson"], DC_MAX_ITERS=case["passes"],
              SORT_INTERVAL=case.get("sort", 0), DTI_RATIO=case.get("dti", 1.0),
              MAGNETIC_FIELD=case.get("magnetic", 0.0))
    plasma = case.get("plasma", "argon")
    if plasma != "default":
        kw.update(HAVE_COLLISIONS=case["kind"] != "phases", SIGMA="ENERGY_DEPENDENT",
                  SIGMA_ELASTIC="ENERGY_DEPENDENT", SIGMA_IONIZATION="ENERGY_DEPENDENT", STEADYSTATE="NO",
                  SIZE_TO_CHECK=2**31 - 1)
    if plasma == "argon":
        kw.update(TEMPERATURE=te, GAS_PRESSURE_TORR=torr)
    elif plasma == "hydrogen":
        te = 3.0
        kw.update(TEMPERATURE=te, ION_MASS_AMU=1.0, THRESHOLD=13.6, SPECIES="HYDROGEN", E_IMPACT_SEE="YES",
                  REFLECTION="YES", BACKSCATTER="YES", NUMBER_TO_INJECT=10)
    else:
        te = 1.5
    length = picgb.make_params(**kw).xlength
    size = 1.0e15 * length * length / n
    return picgb.make_params(E_MACROPARTICLE_SIZE=size, ION_MACROPARTICLE_SIZE=size, **kw), te


def _records(n, length, mass, temperature, seed, profile):
    """n records {x, y, vx, vy, vz, weight} on the GPU: Maxwellian velocities;
    positions uniform in the box, or a Gaussian (sigma = length/4) truncated
    to it"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.empty(n, 6, dtype=torch.float64, device="cuda")
    u = torch.rand(n, 2, generator=g, dtype=torch.float64, device="cuda").clamp_(1e-9, 1.0 - 1e-9)
    if profile == "gaussian":
        half = math.erf(math.sqrt(2.0))
        u = 0.5 + 0.25 * math.sqrt(2.0) * torch.erfinv((2.0 * u - 1.0) * half)
    a[:, 0:2] = length * u
    a[:, 2:5] = math.sqrt(temperature * picgb.CHARGE / mass) * torch.randn(n, 3, generator=g, dtype=torch.float64,
                                                                            device="cuda")
    a[:, 5] = 1.0
    return a


def _pinned(t):
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return p


def _state(p, n, te, seed, profile="uniform"):
    """host records of both species; the ions a little fewer, as a plasma that
    has run for a while holds them"""
    e = _records(n, p.xlength, picgb.ELECTRON_MASS, te, 2 * seed + 1, profile)
    i = _records(n - n // 97, p.xlength, p.ion_mass, 0.026, 2 * seed + 2, profile)
    return _pinned(e), _pinned(i)


def _room(n):
    return n + n // 16 + 8192


class _Held:
    """a run handle and the host buffers its program keeps for it"""

    def __init__(self, p, particles=None):
        self.run = picgb.Run(p)
        self.grid = {w: torch.empty(math.prod(picgb.grid_shape(p, w)), dtype=torch.float64, pin_memory=True)
                     for w in _GRIDS}
        self.records = particles
        if particles:
            # room for what the steps may add; what a dump does not fill stays 0
            self.out = [torch.zeros(_room(r.shape[0]), 6, dtype=torch.float64, pin_memory=True) for r in particles]

    def load(self):
        for s in (0, 1):
            self.run.load_particles_ptr(s, self.records[s].data_ptr(), self.records[s].shape[0])

    def dump(self):
        """both species' records in the program's buffers, and how many"""
        got = [self.run.dump_particles_ptr(s, self.out[s].data_ptr(), self.out[s].shape[0]) for s in (0, 1)]
        return {"e": self.out[0], "i": self.out[1], "n_e": got[0], "n_i": got[1]}

    def grids(self, which):
        r = self.run
        for w in which:
            g = self.grid[w]
            rc = r.lib.pgb_get_grid(r.h, picgb.GRID[w], ctypes.cast(g.data_ptr(), ctypes.POINTER(ctypes.c_double)),
                                    g.numel())
            if rc:
                raise picgb.PicError("pgb_get_grid failed (%d)" % rc, rc)
        return {w: self.grid[w] for w in which}


def _batch_members(case):
    r = random.Random(case["mix"])
    return [{"nodes": r.choice([65, 129, 257]), "particles": _log_int(r, 50000, case["most"]),
             "torr": r.uniform(0.005, 0.05), "te": r.uniform(1.0, 4.0)} for _ in range(case["runs"])]


# ------------------------------------------------------------------- prepare
def _deposit_inputs(case, seed):
    n, nodes = case["particles"], case["nodes"]
    length = 0.01
    a = _records(n, length, picgb.ELECTRON_MASS, 2.0, seed, "gaussian")
    g = torch.Generator(device="cuda").manual_seed(seed + 77)
    k = torch.randint(0, n, (n // 200 + 1,), generator=g, device="cuda")
    a[k, 0] = -0.002 * length          # a few have just left through a wall
    a[k.flip(0)[: n // 400 + 1], 5] = 0.0   # and a few were injected (weight 0)
    if case["order"] == "binned":      # 32 x 32 cells a bin, as a sorted run dumps them
        h = 32.0 * length / (nodes - 1)
        bins = (nodes + 30) // 32
        key = torch.floor(a[:, 1] / h) * bins + torch.floor(a[:, 0] / h)
        a = a[torch.sort(key, stable=True).indices].contiguous()
    return a, length


def _rho_inputs(case, seed):
    """a plasma's charge density: a smooth space charge and the noise of
    about 64 particles a cell, zero outside the walls"""
    n = case["nodes"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda")
    c = 0.6 * torch.rand(2, generator=g, dtype=torch.float64, device="cuda") - 0.3
    smooth = torch.exp(-2.0 * ((s[:, None] - c[0]) ** 2 + (s[None, :] - c[1]) ** 2))
    noise = torch.randn(n, n, generator=g, dtype=torch.float64, device="cuda") / 8.0
    return 1.0e15 * picgb.CHARGE * (0.02 * smooth + 0.1 * noise)


def _fields_params(case, seed):
    w = case["walls"]
    return picgb.make_params(X_NO_OF_CELLS=case["nodes"], TEMPERATURE=2.0, POISSON=case["poisson"],
                             DC_MAX_ITERS=case["passes"], PHI_LEFT=-0.3 * w, PHI_RIGHT=w, PHI_TOP=0.1 * w,
                             PHI_BOTTOM=0.0, PHI_PERIOD=0.02, RAND_SEED=1 + seed % 100003)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "deposit":
        a, length = _deposit_inputs(case, seed)
        q = torch.empty(case["nodes"], case["nodes"], dtype=torch.float64, device="cuda")
        return {"case": case, "lib": picgb.load_library(), "records": a, "q": q, "d": length / (case["nodes"] - 1)}
    if kind == "fields":
        return {"case": case, "held": _Held(_fields_params(case, seed)), "rho": _pinned(_rho_inputs(case, seed))}
    if kind == "batch":
        held = []
        for k, m in enumerate(_batch_members(case)):
            p, te = _params(case, seed + 17 * k, m["nodes"], m["particles"], m["torr"], m["te"])
            held.append(_Held(p, _state(p, m["particles"], te, seed + 1000 * (k + 1))))
        return {"case": case, "held": held}
    if kind == "frame":
        p, te = _params(dict(case, poisson="DST_DC", passes=2, sort=8), seed)
        h = _Held(p, _state(p, case["particles"], te, seed, "gaussian"))
        h.load()
        h.run.initial_boundary()
        h.run.step(4)
        return {"case": case, "held": h, "seed": seed}
    p, te = _params(case, seed)
    profile = "uniform" if case.get("plasma", "argon") == "argon" else "gaussian"
    return {"case": case, "held": _Held(p, _state(p, case["particles"], te, seed, profile))}


# ----------------------------------------------------------------------- run
def _restart(h):
    h.load()
    h.run.set_time_step(0)
    h.run.initial_boundary()


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "deposit":
        a, d = state["records"], state["d"]
        rc = state["lib"].pgb_deposit_static(a.data_ptr(), a.shape[0], case["nodes"], case["nodes"], d, d, -1.6e-13,
                                             state["q"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise picgb.PicError("pgb_deposit_static failed (%d)" % rc, rc)
        return state["q"]
    h = state["held"]
    if kind == "fields":
        r = h.run
        rc = r.lib.pgb_set_rho(r.h, ctypes.cast(state["rho"].data_ptr(), ctypes.POINTER(ctypes.c_double)),
                               state["rho"].numel())
        if rc:
            raise picgb.PicError("pgb_set_rho failed (%d)" % rc, rc)
        r.poisson(3)
        r.efield()
        return h.grids(("phi", "ex", "ey"))
    if kind == "phases":
        r = h.run
        h.load()
        r.set_time_step(0)
        for t in (0, 1):
            if t:
                r.gather_push(0)
                r.gather_push(1)
                r.boundary(picgb.PGB_BOUNDARY_IONS)
                r.boundary(picgb.PGB_BOUNDARY_ELECTRONS)
            r.deposit(1)
            r.deposit(0)
            r.grid_rho()
            r.poisson(t)
            r.efield()
        return dict(h.dump(), grids=h.grids(_GRIDS))
    if kind == "frame":
        c, r = case, h.run
        return [torch.from_numpy(r.render(plot, c["pixels"], c["pixels"], c["points"], state["seed"] % 1000))
                for plot in ("particle_xy", "electron_vx_vy", "phi")]
    if kind == "batch":
        for m in h:
            _restart(m)
        picgb.step_batch([m.run for m in h], case["steps"])
        return [dict(m.dump(), phi=m.grids(("phi",))["phi"]) for m in h]
    _restart(h)
    h.run.step(case["steps"])
    return dict(h.dump(), grids=h.grids(_GRIDS))


# ---------------------------------------------------------------------- work
def _step_work(nodes, n, collisions):
    # a species' state read and written once (x, y, vx, vy and, with
    # collisions, vz; weight and id read), the charge and field grids once
    per = 16 + 16 + 4 + (8 if collisions else 0)
    return 2.0 * n * per + nodes * nodes * (2 * 8 + 8 + 8 + 16), 2.0 * n * 150.0 + nodes * nodes * 200.0


def work(case):
    kind = case["kind"]
    if kind == "deposit":
        return {"bytes": 48.0 * case["particles"] + 8.0 * case["nodes"] ** 2, "flops": 20.0 * case["particles"]}
    if kind == "fields":
        g = float(case["nodes"]) ** 2
        return {"bytes": 8.0 * g * 4, "flops": g * (30.0 * case["passes"] + 50.0)}
    if kind == "frame":
        return {"bytes": 2 * 20.0 * case["particles"] + 9.0 * case["pixels"] ** 2, "flops": 20.0 * case["particles"]}
    members = _batch_members(case) if kind == "batch" else [case]
    steps = 1 if kind == "phases" else case["steps"]
    b = f = 0.0
    for m in members:
        sb, sf = _step_work(m["nodes"], m["particles"], kind == "batch" or case.get("plasma") in ("argon", "hydrogen"))
        b += steps * sb + 2 * 2 * 48.0 * m["particles"]
        f += steps * sf
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------------- exact
def _cic(x, y, w, d, n):
    """cloud-in-cell charge of the particles with 0 < x, y < (n-1) d, rows and
    columns on the edges doubled, corners doubled again (particle.cpp:663-858)"""
    ok = (x > 0) & (y > 0) & (x < (n - 1) * d) & (y < (n - 1) * d)
    xs, ys, w = x[ok] / d, y[ok] / d, w[ok]
    j, k = xs.floor().long(), ys.floor().long()
    a, b = xs - j, ys - k
    q = torch.zeros(n * n, dtype=torch.float64, device=x.device)
    for dk, dj, c in ((0, 0, (1 - a) * (1 - b)), (0, 1, a * (1 - b)), (1, 0, (1 - a) * b), (1, 1, a * b)):
        q.index_add_(0, (k + dk) * n + j + dj, c * w)
    q = q.reshape(n, n)
    q[0] *= 2
    q[-1] *= 2
    q[:, 0] *= 2
    q[:, -1] *= 2
    for r in (0, -1):
        for c in (0, -1):
            q[r, c] *= 2
    return q


def _sine(f):
    """type-I sine transform of the last axis (length N-1)"""
    m = f.shape[-1] + 1
    z = torch.zeros(*f.shape[:-1], 1, dtype=f.dtype, device=f.device)
    return -0.5 * torch.fft.fft(torch.cat([z, f, z, -f.flip(-1)], -1)).imag[..., 1:m]


def _solve(rho, p, t):
    """the 5-point Poisson solution of fields::grid_potential
    (fields.cpp:169-220), converged, and the field of grid_electric_field
    (fields.cpp:230-268)"""
    n = p.x_no_of_cells
    m, d = n - 1, p.xlength / (n - 1)
    right = p.phi_right * math.cos(p.phi_period * t)
    f = -rho / _EPS0
    f[:, 1] -= p.phi_left / (d * d)
    f[:, n - 2] -= right / (d * d)
    f[1, :] -= p.phi_bottom / (d * d)
    f[n - 2, :] -= p.phi_top / (d * d)
    k = torch.arange(1, m, dtype=torch.float64, device=rho.device)
    s = 4.0 * torch.sin(math.pi * k / (2 * m)) ** 2
    c = _sine(_sine(f[1:-1, 1:-1]).T).T * (-(d * d)) / (s[:, None] + s[None, :])
    phi = torch.zeros(n, n, dtype=torch.float64, device=rho.device)
    phi[1:-1, 1:-1] = _sine(_sine(c).T).T * (2.0 / m) ** 2
    phi[:, 0], phi[:, -1] = p.phi_left, right
    phi[0, :], phi[-1, :] = p.phi_bottom, p.phi_top
    ex, ey = torch.zeros_like(phi), torch.zeros_like(phi)
    ex[1:-1, 1:-1] = (phi[1:-1, :-2] - phi[1:-1, 2:]) / (2.0 * d)
    ey[1:-1, 1:-1] = (phi[:-2, 1:-1] - phi[2:, 1:-1]) / (2.0 * d)
    ex[:, 0], ex[:, -1] = 2 * ex[:, 1] - ex[:, 2], 2 * ex[:, -2] - ex[:, -3]
    ey[0, :], ey[-1, :] = 2 * ey[1, :] - ey[2, :], 2 * ey[-2, :] - ey[-3, :]
    return phi, ex, ey


def _padded(e, n):
    """a field grid in its (n+1)*(n+1) buffer with row stride n"""
    out = torch.zeros((n + 1) * (n + 1), dtype=torch.float64, device=e.device)
    out[: n * n] = e.reshape(-1)
    return out


def _push(a, ex, ey, p, dt, q_over_m):
    """gather and push (pic.cl:56-149), both walls absorbing"""
    n = p.x_no_of_cells
    d = p.xlength / (n - 1)
    x, y, vx, vy, vz = (a[:, c] for c in range(5))
    j, k = (x / d).floor().long().clamp(0, n - 1), (y / d).floor().long().clamp(0, n - 1)
    u, v = x / d - j, y / d - k
    exf, eyf = _padded(ex, n), _padded(ey, n)
    base = k * n + j
    corner = ((0, (1 - u) * (1 - v)), (1, u * (1 - v)), (n, (1 - u) * v), (n + 1, u * v))
    px, py = (sum(c * g[base + o] for o, c in corner) for g in (exf, eyf))
    half = 0.5 * dt * q_over_m
    vx, vy = vx + half * px, vy + half * py
    if p.magnetic_field > 0:
        ca, sa = math.cos(p.angle), math.sin(p.angle)
        w = dt * q_over_m * p.magnetic_field
        par, perp = ca * vx + sa * vy, -sa * vx + ca * vy
        vz, perp = -perp * math.sin(w) + math.cos(w) * vz, perp * math.cos(w) + math.sin(w) * vz
        vx, vy = ca * par - sa * perp, sa * par + ca * perp
    vx, vy = vx + half * px, vy + half * py
    x, y = x + dt * vx, y + dt * vy
    keep = (x > -d) & (x < n * d) & (y > -d) & (y < n * d)
    return torch.stack([x, y, vx, vy, vz, a[:, 5]], 1)[keep]


def exact(case, seed):
    kind = case["kind"]
    if kind == "deposit":
        a, length = _deposit_inputs(case, seed)
        d = length / (case["nodes"] - 1)
        return _cic(a[:, 0], a[:, 1], a[:, 5], d, case["nodes"]) * (-1.6e-13 / (d * d))
    if kind == "fields":
        n = case["nodes"]
        phi, ex, ey = _solve(_rho_inputs(case, seed), _fields_params(case, seed), 3)
        return {"phi": phi.reshape(-1), "ex": _padded(ex, n), "ey": _padded(ey, n)}
    if kind == "phases":
        n = case["nodes"]
        p, te = _params(case, seed)
        e, i = (r.cuda() for r in _state(p, case["particles"], te, seed))
        d = p.xlength / (n - 1)
        for t in (0, 1):
            if t:
                e = _push(e, ex, ey, p, p.dt, p.q_over_me)
                i = _push(i, ex, ey, p, p.dti, p.q_over_mi)
            q_e = _cic(e[:, 0], e[:, 1], e[:, 5], d, n) * (p.qce / (d * d))
            q_i = _cic(i[:, 0], i[:, 1], i[:, 5], d, n) * (p.qci / (d * d))
            rho = q_e + q_i
            phi, ex, ey = _solve(rho.clone(), p, t)
        flat = {"q_e": q_e, "q_i": q_i, "rho": rho, "phi": phi}
        grids = {w: g.reshape(-1) for w, g in flat.items()}
        grids.update(ex=_padded(ex, n), ey=_padded(ey, n))
        rec = {}
        for name, a, n0 in (("e", e, case["particles"]), ("i", i, case["particles"] - case["particles"] // 97)):
            rec[name] = torch.zeros(_room(n0), 6, dtype=torch.float64, device=a.device)
            rec[name][: a.shape[0]] = a
        return dict(rec, n_e=e.shape[0], n_i=i.shape[0], grids=grids)
    # plots are bytes, and runs draw from the library's own random streams
    return None
