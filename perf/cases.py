"""The work a user of this package has it do, as cases that can be timed and checked.

Every case is a scene (or several) of jittered 2x2x2-per-cell blocks or beds of sand, snow or elastic material with a smooth
velocity field and a small smooth strain, as a scene in the middle of its run has them, stepped through the public API:

  step    MpmSimulation: a stepping loop's next call on a resident scene (dense or sparse grid, either SVD form, with or without
          the fixed-order P2G, rigid spheres and the semi-implicit sweeps), its positions and velocities read into the caller's
          buffers, left on the device as the render view, or with the whole particle state (C, F, J_p)
  scene   a whole request on one simulation: upload particles and materials, step, read positions and velocities
  batch   MpmGroup: many scenes of uneven size stepped by shared launches through graphs, every scene's positions read
  serve   MpmServer: requests submitted, ticked until all are done, and their positions fetched
  study   MpmSimulation64: the all-FP64 run of a precision study between two of its readings

Sizes are those of this repository's presets, tests and benchmark workloads (the 32^3 and 48^3 presets, the 64^3 cube with
132,651 particles, the 128^3 cube with 1M, the 256^3 scene with 16M, batches of 10k..2M-particle scenes on 32^3..128^3 grids)."""

import math

import numpy as np
import torch

import molla_b200 as mm

SAND, SNOW, ELASTIC = 0, 1, 2
_STRAIN = 4.0e-3  # inside snow's elastic range on average, outside it at the peaks
_engine = None


def engine():
    global _engine
    if _engine is None:
        _engine = mm.Engine(0)
    return _engine


# ---- the cases -------------------------------------------------------------------------------------------------------

_STEP = {"kind": "step", "preset": "unit", "grid": 64, "n": 0, "blocks": 1, "shape": "block", "rows": "elastic", "svd64": False,
         "sticky": False, "implicit": 0, "spheres": 0, "fixed_order": False, "sparse": False, "substeps": 1, "read": "host"}


def _case(**kw):
    return {**_STEP, **kw}


def listed():
    return [
        # An interactive loop on the reference's sand preset: one substep a call, state back on the host each time.
        _case(name="sand patch, one substep", preset="sand", grid=32, n=4_001, shape="bed", rows="sand", substeps=1),
        # Wheel-soil coupling on the calibrated-sand preset (semi-implicit): spheres moved each frame, the reaction read back.
        _case(name="soil bed with wheels", preset="sand_calibrated", grid=48, n=30_000, shape="bed", rows="sand", implicit=3, spheres=4,
              substeps=4, read="view"),
        # Bit-reproducible stepping of a snow scene, its whole state taken for the record.
        _case(name="snow, fixed-order P2G", grid=64, n=100_003, rows="snow", blocks=2, fixed_order=True, substeps=32, read="state"),
        # A small body of material in a large world on sparse storage.
        _case(name="sparse world", grid=256, n=300_000, rows="mixed", blocks=3, sparse=True, substeps=16, read="view"),
        # The 64^3 cube: FP32 state and SVD, sticky walls.
        _case(name="cube 64, FP32", grid=64, n=132_651, sticky=True, substeps=20),
        # The 128^3 cube with the FP64 SVD.
        _case(name="cube 128, FP64 SVD", grid=128, n=1_000_000, sticky=True, svd64=True, substeps=20),
        # A mid-size FP32 scene of several materials, drawn from the device after each frame.
        _case(name="boxes 160, FP32", grid=160, n=3_999_997, rows="mixed", blocks=4, substeps=12, read="view"),
        # The single large scene.
        _case(name="boxes 256, FP64 SVD", grid=256, n=16_000_000, rows="mixed", blocks=4, svd64=True, substeps=16),
        # A whole request with fresh inputs: upload, run, read.
        _case(name="new scene each call", kind="scene", grid=96, n=500_000, rows="snow", blocks=2, substeps=50),
        # Uneven independent scenes in shared launches, graph-replayed.
        {"name": "batch of 24", "kind": "batch", "scenes": 24, "n_lo": 10_000, "n_hi": 600_000, "grid_hi": 128, "substeps": 50},
        # Requests through the continuous-batching loop.
        {"name": "serve 8 requests", "kind": "serve", "scenes": 8, "n_lo": 10_000, "n_hi": 200_000, "grid_hi": 96, "substeps": 60},
        # The precision study's all-FP64 leg between two readings.
        {"name": "all-FP64 cube 64", "kind": "study", "grid": 64, "n": 132_651, "substeps": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 8 + ["scene", "scene", "batch", "serve", "study"])
    if kind in ("batch", "serve"):
        hi = _log(rng, 40_000, 600_000 if kind == "batch" else 200_000)
        return {"kind": kind, "scenes": _log(rng, 2, 32 if kind == "batch" else 10), "n_lo": rng.randint(2_000, 10_000), "n_hi": hi,
                "grid_hi": rng.randint(64, 128), "substeps": rng.randint(20, 80)}
    n = _log(rng, 1_000, 6_000_000 if kind == "step" else 1_000_000 if kind == "scene" else 300_000)
    grid = max(24, math.ceil((n / 8 / 0.2) ** (1 / 3)))
    grid = min(256, max(grid, int(round(grid * rng.uniform(1.0, 1.8)))))
    if kind == "study":
        return {"kind": kind, "grid": min(grid, 128), "n": n, "substeps": rng.randint(10, 100)}
    c = _case(kind=kind, grid=grid, n=n, blocks=rng.randint(1, 4), rows=rng.choice(["sand", "snow", "elastic", "mixed"]),
              svd64=rng.random() < 0.5, sticky=rng.random() < 0.3, substeps=_log(rng, 1, 32), read=rng.choice(["host", "view", "state"] if n <= 500_000 else ["host", "view"]))
    if kind == "scene":
        c["read"] = "host"
        return c
    if n <= 40_000 and rng.random() < 0.6:  # the presets' range
        c.update(preset=rng.choice(["sand", "sand_calibrated", "snow"]), grid=rng.choice([32, 48]), shape="bed", blocks=1, svd64=False,
                 sticky=False)
        c["rows"] = "snow" if c["preset"] == "snow" else "sand"
        if c["preset"] == "sand_calibrated":
            c.update(implicit=rng.randint(1, 4), spheres=rng.randint(0, 4), read="view")
    elif n <= 400_000 and rng.random() < 0.25:
        # on power-of-two grids, where x / dx is exact: on others a particle within rounding of a cell face may stop the fixed order
        c.update(fixed_order=True, grid=32 if grid <= 32 else 64 if grid <= 64 else 128)
    elif rng.random() < 0.25:
        c.update(sparse=True, grid=min(256, grid * 2))
    return c


# ---- inputs ----------------------------------------------------------------------------------------------------------

def _dt(youngs, rho, dx, nu=0.2):
    """dt at a CFL number of 0.4 of the pressure-wave speed."""
    mu, lam = youngs / (2 * (1 + nu)), youngs * nu / ((1 + nu) * (1 - 2 * nu))
    return float(np.float32(0.4 * dx / math.sqrt((lam + 2 * mu) / rho)))


def _config(case):
    """(MpmConfig, material rows as dicts or None, dt) of a step, scene or study case."""
    n, grid = case["n"], case["grid"]
    preset = case.get("preset", "unit")
    if preset != "unit":
        cfg = getattr(mm.MpmConfig, preset)()
        cfg.grid_size, cfg.max_particles = grid, n
        cfg.grid_origin = (-0.5 * grid * cfg.cell_size, 0.0, -0.5 * grid * cfg.cell_size)
        if case["implicit"]:
            cfg.time_step, cfg.jacobi_iters = mm.MpmTimeStep.IMPLICIT, case["implicit"]
        return cfg, None, float(np.float32(1.0 / (1920.0 if preset == "snow" else 480.0)))
    dx, rho, nu = 1.0 / grid, 16.0, 0.2
    elastic = [{"kind": ELASTIC, "youngs": e, "poisson": nu} for e in (2.0e4, 1.0e5)]
    snow = [{"kind": SNOW, "theta_c": 2.5e-2, "theta_s": 7.5e-3, "hardening": 10.0, "youngs": e, "poisson": nu} for e in (4.0e4, 8.0e4)]
    sand = [{"kind": SAND, "friction_angle": math.radians(a), "youngs": 6.0e4, "poisson": nu} for a in (25.0, 35.0)]
    rows = {"elastic": elastic, "snow": snow, "sand": sand, "mixed": [elastic[0], snow[0], sand[0], elastic[1], snow[1]]}[case.get("rows", "elastic")]
    vol = dx ** 3 / 8.0
    sticky = case.get("sticky", True)
    cfg = mm.MpmConfig(grid_size=grid, cell_size=dx, grid_origin=(0.0, 0.0, 0.0), gravity_y=-9.8, youngs=1.0e5, poisson=nu, friction_angle=0.0,
                       boundary_friction=0.0 if sticky else 0.3, particle_mass=rho * vol, particle_volume=vol, max_particles=n,
                       rheology=mm.MpmRheology.from_dict(rows[0]), walls=1 if sticky else 0, boundary_pad=3 if sticky else 0,
                       svd_precision=1 if case.get("svd64") else 0)
    return cfg, rows, _dt(1.0e5, rho, dx)


def _particles(cfg, rows, n, blocks, shape, seed, lift, moving=True):
    """Positions, velocities, C, F (column-major rows of 9), material ids of a scene, on the GPU in FP32."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    u = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    N, dx = cfg.grid_size, cfg.cell_size
    floor = float(cfg.boundary_pad or 2)
    pos, ids = [], []
    blocks = max(1, min(blocks, n))
    for b in range(blocks):
        k = n // blocks + (b < n % blocks)
        if shape == "bed":  # a layer over the middle of the floor
            e = max(2, min(int(1.4 * (N - 2 * floor - 4)), math.ceil(math.sqrt(k / 2))))
            ax, az, ay = e, e, -(-k // (e * e))
        else:
            e = max(1, math.ceil(k ** (1 / 3) - 1e-9))
            ax, az, ay = e, e, -(-k // (e * e))
        i = torch.arange(k, device="cuda")
        q = torch.stack([i % ax, i // (ax * az), (i // ax) % az], 1).double()
        q = (q + 0.5 + (u(k, 3) - 0.5)) * 0.5  # in cells
        at = 0.5 if blocks == 1 else None
        cx, cz = (at, at) if at else ((0.3, 0.7, 0.3, 0.7)[b % 4], (0.3, 0.7, 0.7, 0.3)[b % 4])
        low = torch.tensor([cx * N - 0.25 * ax, floor, cz * N - 0.25 * az], device="cuda").clamp(min=floor).double()
        low[1] += float(u(1)) * lift
        low[0::2] = torch.minimum(low[0::2], torch.tensor(N - floor - 1.0 - 0.5 * max(ax, az), device="cuda").double().clamp(min=floor))
        pos.append(low + q)
        ids.append(torch.full((k,), b % len(rows) if blocks > 1 else 0, device="cuda", dtype=torch.int64))
        if blocks == 1 and len(rows) > 1:  # layers of the materials
            ids[-1] = (q[:, 1] * 2 * len(rows) / max(ay, 1)).long().clamp(0, len(rows) - 1)
        del q
    p = torch.cat(pos)
    del pos
    L = N * dx
    s = p / N  # unit-box coordinates
    x = p * dx + torch.tensor(cfg.grid_origin, device="cuda", dtype=torch.float64)
    vmax = 0.5 * L if cfg.cell_size < 0.04 else 0.3
    drift, twist = (u(3) - 0.5) * vmax, (u(3, 3) - 0.5) * vmax / L
    amp, ph, wave = (0.2 + u(3)) * 0.3 * vmax, u(3) * 6.28, 6.28318 * (1 + torch.floor(2 * u(3)))
    v = drift + (x - x.mean(0)) @ twist.T
    C = twist.T.repeat(len(x), 1, 1)  # C[col][row] = dv_row/dx_col
    for r in range(3):
        c = (r + 1) % 3
        arg = wave[r] * s[:, c] + ph[r]
        v[:, r] += amp[r] * torch.sin(arg)
        C[:, c, r] += amp[r] * wave[r] / L * torch.cos(arg)
    # a small rotation times a smooth strain of a few 1e-3, a little compressive
    E = torch.empty(len(x), 3, 3, device="cuda", dtype=torch.float64)
    a, ph2 = (u(3, 3) - 0.5) * 2 * _STRAIN, u(3, 3) * 6.28
    for c in range(3):
        for r in range(3):
            E[:, c, r] = a[c, r] * torch.sin(6.28318 * s[:, (c + r) % 3] * 2 + ph2[c, r]) - (0.2 * _STRAIN if c == r else 0.0)
    ang = 0.2 * (float(u(1)) - 0.5)
    R = torch.eye(3, device="cuda", dtype=torch.float64)
    R[0, 0] = R[2, 2] = math.cos(ang)
    R[0, 2], R[2, 0] = math.sin(ang), -math.sin(ang)
    F = (torch.eye(3, device="cuda", dtype=torch.float64) + E) @ R.T  # rows are columns of R (I + E)
    out = {"x": x.float(), "ids": torch.cat(ids)}
    if moving:
        out.update(v=v.float(), C=C.reshape(-1, 9).float(), F=F.reshape(-1, 9).float())
    return out


def _spheres(case, seed, frame):
    """Wheels half sunk into the bed, rolling to and fro along x."""
    r = np.random.default_rng(seed)
    cfg, _, dt = _config(case)
    L = cfg.grid_size * cfg.cell_size
    out = []
    for k in range(case["spheres"]):
        z, rad = (k + 0.5) / case["spheres"] * 0.5 * L - 0.25 * L + 0.01 * r.random(), 0.12 + 0.05 * r.random()
        t = frame * case["substeps"] * dt
        w, am, ph = 0.7 + r.random(), 0.2 * L, 6.28 * r.random()
        out.append(((am * math.sin(w * t + ph), 0.2 + 0.05 * r.random(), z), rad, (am * w * math.cos(w * t + ph), 0.0, 0.0)))
    return out


def _many(case, seed):
    """The scenes of a batch or serve case: (config, row dicts, dt, particle count, seed), sizes by the case alone."""
    r = np.random.default_rng([case["scenes"], case["n_lo"], case["n_hi"], case["grid_hi"]])
    out = []
    for k in range(case["scenes"]):
        n = int(round(math.exp(r.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        fit = max(32, math.ceil((n / 8 / 0.2) ** (1 / 3)))
        grid = int(round(math.exp(r.uniform(math.log(min(fit, case["grid_hi"] - 1)), math.log(case["grid_hi"])))))
        n = min(n, int(8 * 0.25 * grid ** 3))
        cfg, rows, dt = _config({"n": n, "grid": grid, "rows": ["elastic", "snow"][k % 2], "sticky": k % 3 == 0})
        out.append((cfg, rows, dt, n, seed * 1000 + k))
    return out


def _pinned(n):
    return torch.empty(n, 3, dtype=torch.float32, pin_memory=True).numpy()


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _host_ids(t):
    return t.to(torch.int32).cpu().numpy().astype(np.uint32)


# ---- the calls -------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "seed": seed}
    if kind in ("batch", "serve"):
        st["scenes"] = []
        for cfg, rows, dt, n, sd in _many(case, seed):
            p = _particles(cfg, rows, n, 1, "block", sd, 0.0, moving=False)
            st["scenes"].append((cfg, rows, _host(p["x"]), _host_ids(p["ids"]), dt))
        if kind == "batch":
            cells = sum((s[0].grid_size ** 3 + 255) // 256 * 256 for s in st["scenes"])
            g = mm.MpmGroup(engine(), len(st["scenes"]), sum(len(s[2]) for s in st["scenes"]), cells)
            st["group"], st["sids"] = g, [g.add_scene(*s) for s in st["scenes"]]
        else:
            st["server"] = mm.MpmServer(engine(), 3 << 30, 64)
        return st
    cfg, rows, dt = _config(case)
    st["dt"] = dt
    if kind == "study":
        p = _particles(cfg, rows, case["n"], 1, "block", seed, 0.0, moving=False)
        sim = mm.MpmSimulation64(engine(), cfg)
        sim.set_particles(p["x"].double().cpu().numpy())
        sim.set_materials(rows, _host_ids(p["ids"]))
        st["sim"] = sim
        return st
    p = _particles(cfg, rows or [None], case["n"], case["blocks"], case["shape"], seed, 0.0 if case["shape"] == "bed" else 3.0)
    if case["sparse"]:
        sim = mm.MpmSimulation.new_sparse(engine(), cfg, ((cfg.grid_size + 3) // 4) ** 3 // 4)
    else:
        sim = mm.MpmSimulation.new(engine(), cfg)
    st["sim"], st["pos"], st["vel"] = sim, _pinned(case["n"]), _pinned(case["n"])
    if kind == "scene":
        st["x"], st["v"] = (torch.empty(case["n"], 3, pin_memory=True).copy_(p[k]).numpy() for k in ("x", "v"))
        st["ids"], st["rows"] = _host_ids(p["ids"]), rows
        return st
    sim.set_particles(_host(p["x"]), _host(p["v"]))
    if rows:
        sim.set_materials(rows, _host_ids(p["ids"]))
    sim.write_particle_state(_host(p["C"]), _host(p["F"]))
    if case["fixed_order"]:
        sim.prepare_particle_tile_ordering(case["n"])
        sim.set_particle_tile_ordering(True)
        sim.prepare_deterministic_p2g()
        sim.set_deterministic_p2g(True)
    if case["spheres"]:
        st["frame"] = 0
    if case["read"] == "view":
        st["view"] = torch.as_tensor(sim.particle_render_view(), device="cuda")
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "batch":
        st["group"].step_graph(case["substeps"])
        return [st["group"].read_positions(s) for s in st["sids"]]
    if kind == "serve":
        srv = st["server"]
        tickets = [srv.submit(*s, steps=case["substeps"] + 7 * (k % 3)) for k, s in enumerate(st["scenes"])]
        out = [None] * len(tickets)
        while any(o is None for o in out):
            srv.run(1, 20)
            for k, t in enumerate(tickets):
                if out[k] is None:
                    state, pos = srv.poll(t)
                    out[k] = pos if state >= 2 else None
        return out
    sim = st["sim"]
    if kind == "study":
        sim.step_n(st["dt"], case["substeps"])
        return sim.read_state()
    if kind == "scene":
        sim.set_particles(st["x"], st["v"])
        sim.set_materials(st["rows"], st["ids"])
    if case["spheres"]:
        sim.set_rigid_spheres(_spheres(case, st["seed"], st["frame"]))
        st["frame"] += 1
    sim.step_n(st["dt"], case["substeps"])
    if case["spheres"]:
        return [st["view"], np.array(sim.read_rigid_wrenches())]
    if case["read"] == "view":
        return st["view"]
    out = [sim.read_positions(st["pos"]), sim.read_velocities(st["vel"])]
    return out + list(sim.read_particle_state()) if case["read"] == "state" else out


def work(case):
    """Each substep reads and writes a particle's x, F and J_p and reads its mass, volume and material (116 B; twice that in
    FP64) and takes a node's mass and momentum, and its velocity, through memory once (8 particles a node); about 1500
    operations a particle-substep (two 27-node loops, an SVD, a return mapping and the stress)."""
    if case["kind"] in ("batch", "serve"):
        ps = sum(s[3] for s in _many(case, 0)) * (case["substeps"] + (7 if case["kind"] == "serve" else 0))
        return {"bytes": ps * (116 + 6), "flops": ps * 1500}
    ps = case["n"] * case["substeps"]
    wide = 2 if case["kind"] == "study" else 1
    return {"bytes": wide * ps * (116 + 6), "flops": ps * 1500}


def tolerance(case):
    """About four times what another order of the FP32 grid sums, or the step in 64 bits, was seen to differ by.  Positions
    differ by their own rounding (1e-7..4e-7).  Velocities carry the stress, which the FP32 SVD form has to a few FP32 ulps of
    F over a strain of 1e-3 (up to 4e-4 after 50 substeps), the FP64 SVD form from F's own rounding (up to 4e-5)."""
    if case["kind"] == "study":
        return {"rel": 1e-10, "max": 1e-8}
    if case["kind"] in ("batch", "serve") or case["read"] == "view" and not case["spheres"]:
        return {"rel": 2e-6, "max": 1e-4}
    return {"rel": 2e-4, "max": 1e-2} if case["svd64"] else {"rel": 2e-3, "max": 1e-1}


# ---- the step in 64 bits ---------------------------------------------------------------------------------------------

def _jacobi_svd(F):
    """Singular values and vectors of F (lists of 3x3 entries F[r][c], FP64) by Jacobi on F^T F: (u, s, v), u[r][i]."""
    A = [[sum(F[k][i] * F[k][j] for k in range(3)) for j in range(3)] for i in range(3)]
    one, zero = torch.ones_like(F[0][0]), torch.zeros_like(F[0][0])
    V = [[one.clone() if i == j else zero.clone() for j in range(3)] for i in range(3)]
    for _ in range(6):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            k = 3 - p - q
            d, e = A[q][q] - A[p][p], 2.0 * A[p][q]
            h = d.abs() + torch.sqrt(d * d + e * e)
            t = torch.where(h > 0, torch.where(d >= 0, e, -e) / torch.where(h > 0, h, one), zero)
            c = 1.0 / torch.sqrt(1.0 + t * t)
            s = t * c
            A[p][p], A[q][q] = A[p][p] - t * A[p][q], A[q][q] + t * A[p][q]
            A[p][q] = A[q][p] = zero
            kp, kq = A[k][p], A[k][q]
            A[k][p] = A[p][k] = c * kp - s * kq
            A[k][q] = A[q][k] = s * kp + c * kq
            for r in range(3):
                V[r][p], V[r][q] = c * V[r][p] - s * V[r][q], s * V[r][p] + c * V[r][q]
    FV = [[sum(F[r][k] * V[k][i] for k in range(3)) for i in range(3)] for r in range(3)]
    S = [torch.sqrt(sum(FV[r][i] ** 2 for r in range(3))) for i in range(3)]  # F stays near a rotation here: det F > 0
    return [[FV[r][i] / S[i] for i in range(3)] for r in range(3)], S, V


def _exact_steps(cfg, rows, dt, substeps, x, v, C, F, ids, spheres=()):
    """The explicit MLS-MPM substep (quadratic B-splines, APIC, fixed-corotated stress, wall rules, return mappings, the rigid
    imprint and the semi-implicit sweeps) in FP64.  C, F as [n, col, row].  Returns x, v, C, F, J_p and the last substep's wrenches."""
    f32 = lambda a: float(np.float32(a))  # noqa: E731
    N, dt = cfg.grid_size, f32(dt)
    dx = f32(cfg.cell_size)
    inv = f32(1.0 / np.float32(cfg.cell_size))
    o = [f32(a) for a in cfg.grid_origin]
    pad, fric, mass, vol = cfg.boundary_pad or 2, f32(cfg.boundary_friction), f32(cfg.particle_mass), f32(cfg.particle_volume)
    dev, n = x.device, len(x)
    lo = [f32(np.float32(a) + np.float32(pad) * np.float32(dx)) for a in o]
    hi = [f32(np.float32(a) + np.float32(N - pad - 1) * np.float32(dx)) for a in o]
    rh = [r if r is not None else {k: getattr(cfg.rheology, k) for k in ("kind", "friction_angle", "theta_c", "theta_s", "hardening")} for r in (rows or [None])]

    def per(f):
        return torch.tensor([f32(f(r)) for r in rh], device=dev, dtype=torch.float64)[ids]

    E, nu = per(lambda r: r.get("youngs") or cfg.youngs), per(lambda r: r["poisson"] if r.get("youngs") else cfg.poisson)
    mu, lam = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
    kind = per(lambda r: r["kind"])
    hard, tc, ts = (per(lambda r, k=k: r.get(k, 0.0)) for k in ("hardening", "theta_c", "theta_s"))
    alpha = per(lambda r: math.sqrt(2 / 3) * 2 * math.sin(f32(r.get("friction_angle", 0.0))) / (3 - math.sin(f32(r.get("friction_angle", 0.0)))))
    kappa = (3 * lam + 2 * mu) / (2 * mu)
    kinds = {int(r["kind"]) for r in rh}
    x, v, jp = x.double(), v.double(), torch.zeros(n, device=dev, dtype=torch.float64)
    C = [[C[:, c, r].double() for c in range(3)] for r in range(3)]
    F = [[F[:, c, r].double() for c in range(3)] for r in range(3)]
    usv, wrench = None, np.zeros((len(spheres), 2, 3))
    ar = torch.arange(N, device=dev)
    node = [(ar.double() * dx + o[a]) for a in range(3)]
    shape = [(1, 1, N), (1, N, 1), (N, 1, 1)]  # x fastest

    def stencil():
        xp = (x - torch.tensor(o, device=dev, dtype=torch.float64)) * inv
        b = torch.floor(xp - 0.5)
        fx = xp - b
        w = [0.5 * (1.5 - fx) ** 2, 0.75 - (fx - 1.0) ** 2, 0.5 * (fx - 0.5) ** 2]
        b = b.long()
        return b[:, 0] + N * (b[:, 1] + N * b[:, 2]), fx, w

    for _ in range(substeps):
        # scatter
        U, S, V = usv or _jacobi_svd(F)
        h = torch.ones_like(jp)
        h = torch.where(kind == SNOW, torch.exp((-hard * jp).clamp(-3, 3)), h)
        h = torch.where(kind == SAND, torch.exp(jp.clamp(-3, 3)), h)
        Sc = [a.clamp(0.1, 10.0) for a in S]
        J = Sc[0] * Sc[1] * Sc[2]
        tau = [2 * mu * h * (a - 1) * a + lam * h * (J - 1) * J for a in Sc]
        k = -dt * vol * 4.0 * inv * inv
        B = [[mass * C[r][c] + k * sum(U[r][i] * tau[i] * U[c][i] for i in range(3)) for c in range(3)] for r in range(3)]
        base, fx, w = stencil()
        grid = torch.zeros(N ** 3, 4, device=dev, dtype=torch.float64)
        for q in range(27):
            i, j, l = q // 9, q // 3 % 3, q % 3
            d = [(i - fx[:, 0]) * dx, (j - fx[:, 1]) * dx, (l - fx[:, 2]) * dx]
            wt = w[i][:, 0] * w[j][:, 1] * w[l][:, 2]
            val = torch.stack([wt * mass] + [wt * (mass * v[:, r] + B[r][0] * d[0] + B[r][1] * d[1] + B[r][2] * d[2]) for r in range(3)], 1)
            grid.index_add_(0, base + i + N * (j + N * l), val)
        del B, tau, val
        # grid
        gm = grid[:, 0].reshape(N, N, N)
        mom = [grid[:, 1 + a].reshape(N, N, N) for a in range(3)]
        rigid = torch.zeros_like(gm, dtype=torch.bool)
        wrench[:] = 0.0
        fdt = 1.0 / max(dt, 1e-6)
        arms = []
        for s, (c, rad, sv) in enumerate(spheres):
            c, rad, sv = [f32(a) for a in c], f32(rad), [f32(a) for a in sv]
            arm = [(node[a] - c[a]).reshape(shape[a]) for a in range(3)]
            dist = torch.sqrt(arm[0] ** 2 + arm[1] ** 2 + arm[2] ** 2)
            arms.append((arm, dist, rad, sv))
            inside = (dist < rad) & ~rigid
            f = [torch.where(inside & (gm > 1e-9), -(gm * sv[a] - mom[a]) * fdt, torch.zeros_like(gm)) for a in range(3)]
            for a in range(3):
                wrench[s, 0, a] += float(f[a].sum())
                wrench[s, 1, a] += float((arm[(a + 1) % 3] * f[(a + 2) % 3] - arm[(a + 2) % 3] * f[(a + 1) % 3]).sum())
            gm = torch.where(inside, torch.full_like(gm, 1e6), gm)
            mom = [torch.where(inside, torch.full_like(gm, 1e6 * sv[a]), mom[a]) for a in range(3)]
            rigid |= inside
        live = gm > 1e-9
        den = torch.where(live, gm, torch.ones_like(gm))
        gv = [torch.where(live, mom[a] / den, torch.zeros_like(gm)) for a in range(3)]
        gv[1] = torch.where(live & ~rigid, gv[1] + dt * f32(cfg.gravity_y), gv[1])
        free = live & ~rigid
        if cfg.walls:
            edge = torch.zeros_like(live)
            for a in range(3):
                edge = edge | ((ar < pad) | (ar >= N - pad)).reshape(shape[a])
            gv = [torch.where(edge & free, torch.zeros_like(gm), g) for g in gv]
        else:
            for a in range(3):
                for side, clip in (((ar < pad), lambda t: t.clamp(min=0.0)), ((ar >= N - pad), lambda t: t.clamp(max=0.0))):
                    at = side.reshape(shape[a]) & free
                    gv = [torch.where(at, clip(g) if b == a else g * fric, g) for b, g in enumerate(gv)]
        for _s in range(cfg.jacobi_iters if cfg.time_step else 0):
            cnt, tot = torch.zeros_like(gm), [torch.zeros_like(gm) for _ in range(3)]
            for dim in range(3):
                for step in (1, -1):
                    to = [slice(None)] * 3
                    fr = [slice(None)] * 3
                    to[dim], fr[dim] = (slice(0, N - 1), slice(1, N)) if step == 1 else (slice(1, N), slice(0, N - 1))
                    cnt[tuple(to)] += live[tuple(fr)].double()
                    for a in range(3):
                        tot[a][tuple(to)] += torch.where(live, gv[a], torch.zeros_like(gm))[tuple(fr)]
            al = dt * dt * gm * (f32(cfg.youngs) / 1500.0) * inv * inv
            mean = [torch.where(cnt > 0, tot[a] / cnt.clamp(min=1), gv[a]) for a in range(3)]
            gv = [torch.where(free, (gm * gv[a] + al * mean[a]) / torch.where(free, gm + al, torch.ones_like(gm)), gv[a]) for a in range(3)]
        for s, (arm, dist, rad, sv) in enumerate(arms):
            wq = torch.where(dist > rad, (1.0 - (dist - rad) / dx).clamp(min=0.0), torch.ones_like(gm))
            at = free & (dist <= rad + dx)
            f = [torch.where(at, -(gm * wq * fdt) * (sv[a] - gv[a]), torch.zeros_like(gm)) for a in range(3)]
            for a in range(3):
                wrench[s, 0, a] += float(f[a].sum())
                wrench[s, 1, a] += float((arm[(a + 1) % 3] * f[(a + 2) % 3] - arm[(a + 2) % 3] * f[(a + 1) % 3]).sum())
        gvel = torch.stack([g.reshape(-1) for g in gv], 1)
        del grid, gm, mom, gv, den, live, free, rigid
        # gather
        nv = torch.zeros_like(v)
        C = [[torch.zeros_like(jp) for _ in range(3)] for _ in range(3)]
        for q in range(27):
            i, j, l = q // 9, q // 3 % 3, q % 3
            g = gvel[base + i + N * (j + N * l)] * (w[i][:, 0] * w[j][:, 1] * w[l][:, 2]).unsqueeze(1)
            nv += g
            d = [(i - fx[:, 0]) * dx, (j - fx[:, 1]) * dx, (l - fx[:, 2]) * dx]
            for c in range(3):
                for r in range(3):
                    C[r][c] += 4.0 * inv * inv * g[:, r] * d[c]
        del g, d, gvel, w, fx, base
        v = nv
        x = x + dt * v
        for a in range(3):
            v[:, a] = torch.where((x[:, a] < lo[a]) | (x[:, a] > hi[a]), torch.zeros_like(jp), v[:, a])
            x[:, a].clamp_(lo[a], hi[a])
        F = [[F[r][c] + dt * sum(C[r][m] * F[m][c] for m in range(3)) for c in range(3)] for r in range(3)]
        # return mapping
        U, S, V = _jacobi_svd(F)
        T = [a.clone() for a in S]
        if SNOW in kinds:
            sn = kind == SNOW
            T = [torch.where(sn, torch.minimum(torch.maximum(a, 1 - tc), 1 + ts), a) for a in T]
            dl = torch.log(S[0] * S[1] * S[2]) - torch.log(T[0] * T[1] * T[2])
            jp = torch.where(sn, (jp + dl).clamp(-5, 5), jp)
        if SAND in kinds:
            sd = kind == SAND
            ep = [torch.log(a) for a in S]
            tr = ep[0] + ep[1] + ep[2]
            de = [a - tr / 3 for a in ep]
            dn = torch.sqrt(de[0] ** 2 + de[1] ** 2 + de[2] ** 2)
            fy = dn + kappa * tr * alpha
            rc = (-alpha * kappa * tr).clamp(min=0.0)
            out, flow = sd & (tr > 0), sd & (tr <= 0) & (dn > 0) & (fy > 0)
            sc = rc / torch.where(dn > 0, dn, torch.ones_like(dn))
            T = [torch.where(out, torch.ones_like(a), torch.where(flow, torch.exp(de[i] * sc + tr / 3), a)) for i, a in enumerate(T)]
            dq = torch.where(out, torch.sqrt(ep[0] ** 2 + ep[1] ** 2 + ep[2] ** 2), torch.where(flow, fy, torch.zeros_like(fy)))
            jp = torch.where(sd, (jp + dq).clamp(0, 5), jp)
        S = [a.clamp(0.05, 20.0) for a in T]
        F = [[sum(U[r][i] * S[i] * V[c][i] for i in range(3)) for c in range(3)] for r in range(3)]
        usv = (U, S, V)
    flat = lambda M: torch.stack([M[r][c] for c in range(3) for r in range(3)], 1)  # noqa: E731
    return x, v, flat(C), flat(F), jp, wrench


def _from_rest(p):
    n = len(p["x"])
    eye = torch.eye(3, device="cuda").reshape(1, 3, 3).repeat(n, 1, 1)
    return p["x"], torch.zeros_like(p["x"]), torch.zeros(n, 3, 3, device="cuda"), eye, p["ids"]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        out = []
        for k, (cfg, rows, dt, n, sd) in enumerate(_many(case, seed)):
            if k >= 6:  # the others are left out for time
                out.append(None)
                continue
            p = _particles(cfg, rows, n, 1, "block", sd, 0.0, moving=False)
            steps = case["substeps"] + (7 * (k % 3) if kind == "serve" else 0)
            out.append(_exact_steps(cfg, rows, dt, steps, *_from_rest(p))[0])
        return out
    cfg, rows, dt = _config(case)
    if kind == "study":
        p = _particles(cfg, rows, case["n"], 1, "block", seed, 0.0, moving=False)
        x, v, _, F, _, _ = _exact_steps(cfg, rows, dt, case["substeps"], *_from_rest(p))
        return x, v, F
    p = _particles(cfg, rows or [None], case["n"], case["blocks"], case["shape"], seed, 0.0 if case["shape"] == "bed" else 3.0)
    if kind == "scene":
        start = (p["x"], p["v"], *_from_rest(p)[2:])
    else:
        start = (p["x"], p["v"], p["C"].reshape(-1, 3, 3), p["F"].reshape(-1, 3, 3), p["ids"])
    sph = _spheres(case, seed, 0)
    x, v, C, F, jp, wr = _exact_steps(cfg, rows, dt, case["substeps"], *start, spheres=sph)
    view = torch.cat([x, torch.zeros_like(x[:, :1])], 1)
    if sph:
        return [view, wr]
    return {"view": view, "host": [x, v], "state": [x, v, C, F, jp]}[case["read"]]
