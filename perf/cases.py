"""Performance cases: the work that users of the framework have it do, through its public entry points.

Kinds of case:

  fluid2  a World2 advanced by `steps` steps from a given state (a scene restart, an episode, a parameter
          study): the state is set, the world stepped, the particles read back. `io` = "host" exchanges the
          state through host arrays and steps frame by frame (World2.step), as an engine that draws every
          frame does; "device" keeps it on the GPU (set_state_device, step_n, get_state_device).
  batch2  many independent scenes of uneven size advanced together (Batch.step).
  fluid3  the same for a World3, whose state is exchanged through host arrays (set_state, step_n, particles).
  closure coarse steps of the learned closure on a World2 (World2.closure_step), tolerance arithmetic.
  train   Adam iterations of the closure network from given parameters (Mlp.train).

`mode` is the arithmetic: "exact" (the default of a world) or "tolerance". `terms` "plain" is the SI water of
the dam-break scenes (Tait, XSPH), "unit" the reference's default config (linear equation of state), "all" two
phases with artificial viscosity, cohesion, wall friction, CFL substeps and a round obstacle.

Particles sit on a jittered lattice, as the scenes of phi_eng_b200.scenes do, and move with a smooth field plus
particle-scale noise, so neighbour counts and velocities are those of a flow under way.
"""
import math
import os

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EPS = 1e-6


def listed():
    return [
        # the reference's example scene (8 x 12 particles in the unit tank), frame by frame with host read-back:
        # the smallest call, where latency is everything
        {"name": "tank_96", "kind": "fluid2", "nx": 8, "ny": 12, "terms": "unit", "mode": "exact", "steps": 20,
         "io": "host"},
        # the 4,096-particle dam break, the reference's particle cap
        {"name": "dam_4k", "kind": "fluid2", "nx": 64, "ny": 64, "terms": "plain", "mode": "exact", "steps": 50,
         "io": "device"},
        # every optional pair term, two phases and CFL substeps at a ragged size under the cap
        {"name": "two_phase_4k", "kind": "fluid2", "nx": 67, "ny": 59, "terms": "all", "mode": "exact", "steps": 10,
         "io": "device"},
        # a mid-size scene of odd extents in the tolerance mode
        {"name": "dam_32k_tol", "kind": "fluid2", "nx": 207, "ny": 157, "terms": "plain", "mode": "tolerance",
         "steps": 20, "io": "device"},
        # a large scene in the default arithmetic
        {"name": "dam_256k", "kind": "fluid2", "nx": 512, "ny": 512, "terms": "plain", "mode": "exact", "steps": 10,
         "io": "device"},
        # the 1,048,576-particle dam break, the benchmark's default workload
        {"name": "dam_1m_tol", "kind": "fluid2", "nx": 1024, "ny": 1024, "terms": "plain", "mode": "tolerance",
         "steps": 10, "io": "device"},
        # the 512-scene batch, 1,024 to 32,768 particles a scene
        {"name": "batch_512_tol", "kind": "batch2", "scenes": 512, "n_min": 1024, "n_max": 32768,
         "mode": "tolerance", "steps": 4},
        # 3D at the reference's particle cap
        {"name": "dam3d_4k", "kind": "fluid3", "nx": 16, "ny": 16, "nz": 16, "mode": "exact", "steps": 30},
        # 3D, a ragged mid-size block in the default arithmetic
        {"name": "dam3d_80k", "kind": "fluid3", "nx": 47, "ny": 41, "nz": 42, "mode": "exact", "steps": 30},
        # 3D, the benchmark's 100^3 block
        {"name": "dam3d_1m_tol", "kind": "fluid3", "nx": 100, "ny": 100, "nz": 100, "mode": "tolerance",
         "steps": 50},
        # the learned closure on the 1,048,576-particle dam break: one block of eight coarse steps
        {"name": "closure_1m", "kind": "closure", "nx": 1024, "ny": 1024, "steps": 8},
        # training of the closure network at its own batch size
        {"name": "train_64k", "kind": "train", "pairs": 1 << 20, "batch": 65536, "iters": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fluid2", "fluid2", "fluid2", "batch2", "fluid3", "fluid3", "closure", "train"])
    mode = rng.choice(["exact", "tolerance"])
    if kind == "fluid2":
        terms = rng.choice(["plain", "plain", "unit", "all"])
        n = _log_int(rng, 64, 6000 if terms != "plain" else 1 << 20)
        nx = max(4, int(round(math.sqrt(n * rng.uniform(0.5, 2.0)))))
        ny = max(4, min(n // nx, (1 << 20) // nx))
        return {"kind": kind, "nx": nx, "ny": ny, "terms": terms, "mode": mode,
                "steps": rng.randint(4, 10 if n > 100000 else 40),
                "io": rng.choice(["host", "device"]) if n < 10000 else "device"}
    if kind == "batch2":
        n_min = _log_int(rng, 64, 2048)
        return {"kind": kind, "scenes": _log_int(rng, 2, 256), "n_min": n_min, "n_max": n_min * rng.randint(2, 16),
                "mode": mode, "steps": rng.randint(2, 8)}
    if kind == "fluid3":
        n = _log_int(rng, 64, 500000)
        nx = max(3, int(round(n ** (1 / 3) * rng.uniform(0.7, 1.4))))
        ny = max(3, int(round(math.sqrt(n / nx) * rng.uniform(0.8, 1.25))))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": max(3, n // (nx * ny)), "mode": mode,
                "steps": rng.randint(10, 30)}
    if kind == "closure":
        n = _log_int(rng, 4096, 1 << 20)
        nx = max(32, int(round(math.sqrt(n * rng.uniform(0.5, 2.0)))))
        return {"kind": kind, "nx": nx, "ny": max(32, min(n // nx, (1 << 20) // nx)), "steps": rng.randint(2, 8)}
    return {"kind": kind, "pairs": _log_int(rng, 50000, 1 << 20), "batch": 128 * _log_int(rng, 8, 512),
            "iters": rng.randint(16, 64)}


# ---------------------------------------------------------------- inputs
def _f32(v):
    return float(np.float32(v))


def _config(case):
    """The fluid config of a case as plain values (f32-exact), its dt and its geometry unit (the spacing)."""
    kind = case["kind"]
    if kind == "fluid3" or case.get("terms") == "unit":
        c = dict(particle_mass=0.0625, rest_density=1.0, smoothing_length=0.5, stiffness=100.0, gamma=1.0,
                 artificial_viscosity=0.0, surface_tension=0.0, cfl=0.0, max_substeps=1, viscosity=0.3, drag=4.0,
                 wall_friction=0.0, max_velocity=30.0, particle_radius=0.125, phase_count=1)
        rest, mass, s, dt = [1.0] * 4, [0.0625] * 4, 0.25, 1.0 / 60.0
    else:
        s = 0.001 if kind == "closure" or case.get("nx", 0) * case.get("ny", 0) >= 200000 else 0.01
        c = dict(particle_mass=s * s, rest_density=1.0, smoothing_length=2.0 * s, stiffness=100.0, gamma=7.0,
                 artificial_viscosity=0.0, surface_tension=0.0, cfl=0.0, max_substeps=1, viscosity=0.3, drag=4.0,
                 wall_friction=0.0, max_velocity=30.0, particle_radius=0.5 * s, phase_count=1)
        rest, mass = [1.0] * 4, [s * s] * 4
        dt = 0.4 * _f32(2.0 * s) / math.sqrt(700.0)
        if case.get("terms") == "all":
            c.update(artificial_viscosity=0.1, surface_tension=20.0, wall_friction=0.2, cfl=0.4, max_substeps=4,
                     phase_count=2)
            rest[1], mass[1] = 0.5, 0.5 * s * s
            dt *= 1.7  # two CFL substeps
    c = {k: (v if k in ("phase_count", "max_substeps") else _f32(v)) for k, v in c.items()}
    return c, [_f32(v) for v in rest], [_f32(v) for v in mass], _f32(dt), s


def _ffi(cfg, rest, mass, into):
    for k, v in cfg.items():
        setattr(into, k, v)
    for k in range(4):
        into.phase_rest_density[k] = rest[k]
        into.phase_mass[k] = mass[k]
    return into


def _block2(rng, nx, ny, s, calm):
    """A moving block of fluid: jittered lattice, smooth velocity field plus noise, f32 [n][4]."""
    n = nx * ny
    iy, ix = np.divmod(np.arange(n), nx)
    q = np.empty((n, 4), np.float32)
    jit = 0.01 if calm else 0.06
    q[:, 0] = (ix + 0.5 + jit * (2.0 * rng.random(n) - 1.0)) * s
    q[:, 1] = (iy + 0.5 + jit * (2.0 * rng.random(n) - 1.0)) * s
    if calm:
        q[:, 2:] = 0.0
    else:
        L = max(nx, ny) * s
        a, b = rng.uniform(0.2, 0.6, 2)
        q[:, 2] = a * np.sin(3.0 * q[:, 1] / L) + 0.02 * rng.standard_normal(n)
        q[:, 3] = -b * np.sin(2.0 * q[:, 0] / L) + 0.02 * rng.standard_normal(n)
    return q


def _walls2(width, height, t):
    return [(0.5 * width, -0.5 * t, 0.5 * width + t, 0.5 * t),
            (-0.5 * t, 0.5 * height, 0.5 * t, 0.5 * height + t),
            (width + 0.5 * t, 0.5 * height, 0.5 * t, 0.5 * height + t),
            (0.5 * width, height + 0.5 * t, 0.5 * width + t, 0.5 * t)]


def _scene2(case, seed):
    """State, phases, boxes, circles and gravity of a single 2D world."""
    rng = np.random.default_rng([seed, 2])
    s = _config(case)[4]
    nx, ny = case["nx"], case["ny"]
    q = _block2(rng, nx, ny, s, case["kind"] == "closure")
    W, H, t = 2.5 * nx * s, 1.5 * ny * s, max(0.1, 4 * s)
    ph, circles = None, []
    if case.get("terms") == "all":
        ph = (np.arange(nx * ny) // nx >= ny // 2).astype(np.uint8)
        circles = [(1.5 * nx * s, 0.0, 0.2 * nx * s)]
    return q, ph, _walls2(W, H, t), circles, (0.0, -9.81)


def _batch_shapes(case, seed):
    rng = np.random.default_rng([seed, 3])
    out = []
    for _ in range(case["scenes"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        nx = max(4, int(round(math.sqrt(n * rng.uniform(0.5, 2.0)))))
        th = math.radians(rng.uniform(-15.0, 15.0))
        out.append((n, nx, -(-n // nx), (9.81 * math.sin(th), -9.81 * math.cos(th))))
    return out


def _batch_scenes(case, seed):
    """[(state, boxes, gravity)] of the batch's scenes. The sizes come from a fixed seed (a batch has one
    configuration for every seed), the states from this one."""
    s, rng, out = 0.01, np.random.default_rng([seed, 4]), []
    for n, nx, ny, g in _batch_shapes(case, 1):
        out.append((_block2(rng, nx, ny, s, False)[:n], _walls2(2.5 * nx * s, 1.5 * ny * s, 0.1), g))
    return out


def _scene3(case, seed):
    rng = np.random.default_rng([seed, 5])
    nx, ny, nz, s = case["nx"], case["ny"], case["nz"], 0.25
    n = nx * ny * nz
    i, j, k = np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij")
    p = np.stack([i, j, k], -1).reshape(n, 3) + 0.5 + 0.04 * (2.0 * rng.random((n, 3)) - 1.0)
    q = np.zeros((n, 6), np.float32)
    q[:, :3] = p * s
    q[:, 3:] = 0.3 * np.sin(2.0 * p[:, ::-1] / max(nx, ny, nz)) + 0.02 * rng.standard_normal((n, 3))
    X, Y, Z, t = 2.5 * nx * s, 1.5 * ny * s, 1.5 * nz * s, 0.5
    boxes = [(X / 2, -t, Z / 2, X / 2 + t, t, Z / 2 + t), (-t, Y / 2, Z / 2, t, Y / 2, Z / 2 + t),
             (X + t, Y / 2, Z / 2, t, Y / 2, Z / 2 + t), (X / 2, Y / 2, -t, X / 2, Y / 2, t),
             (X / 2, Y / 2, Z + t, X / 2, Y / 2, t)]
    return q, boxes


def _pairs(case, seed):
    """Training pairs shaped like the closure's: unit-scale features, targets a smooth map of two of them."""
    g = torch.Generator().manual_seed(int(seed) * 2 + 1)
    x = torch.randn((case["pairs"], 16), generator=g)
    t = 0.05 * torch.stack([torch.tanh(x[:, 0] + 0.5 * x[:, 13]), torch.tanh(x[:, 1] - 0.5 * x[:, 14])], 1)
    w = torch.empty(16 * 64 + 64 + 64 * 64 + 64 + 64 * 2 + 2)
    at = 0
    for rows, cols in ((64, 16), (64, 64), (2, 64)):
        w[at:at + rows * cols] = torch.randn(rows * cols, generator=g) / math.sqrt(cols)
        w[at + rows * cols:at + rows * cols + rows] = 0.1 * torch.randn(rows, generator=g)
        at += rows * cols + rows
    norm = torch.cat([torch.zeros(16), torch.ones(16), torch.tensor([0.05, 0.05])])
    return x, t, w.numpy(), norm.numpy()


# ---------------------------------------------------------------- prepare / run
def _world2(case, q, ph, boxes, circles, gravity):
    from phi_eng_b200 import _abi
    from phi_eng_b200.world import Box, Circle, World2

    cfg, rest, mass, _, _ = _config(case)
    w = World2()
    w.gravity = gravity
    for px, py, hx, hy in boxes:
        w.add_static_body((px, py), Box(hx, hy))
    for px, py, r in circles:
        w.add_static_body((px, py), Circle(r))
    w.fluid.config = _ffi(cfg, rest, mass, _abi.default_config())
    w.fluid.set_cap(max(4096, len(q)))
    got = w.fluid.add_particles(q[:, :2]) if ph is None else w.fluid.add_particles_phase(q[:, :2], ph)
    if got != len(q):
        raise RuntimeError(f"added {got} of {len(q)} particles")
    return w


def _precision(w, mode):
    from phi_eng_b200 import _abi

    w.precision = _abi.TOLERANCE if mode == "tolerance" else _abi.EXACT


def _device_io(w, q):
    """Device copies of the start state and room for the result, the world on torch's stream, as a program
    that reads the result with torch has it."""
    from phi_eng_b200.closure import torch_stream_handle

    w.set_stream(torch_stream_handle())
    x0 = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    out = torch.empty_like(x0)
    torch.cuda.synchronize()
    w.set_state_device(x0.data_ptr(), len(q))
    w.sync()
    return x0, out


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case, "dt": _config(case)[3] if kind != "train" else 0.0}
    if kind in ("fluid2", "closure"):
        q, ph, boxes, circles, g = _scene2(case, seed)
        w = _world2(case, q, ph, boxes, circles, g)
        _precision(w, case.get("mode", "tolerance"))
        st.update(w=w, n=len(q))
        if case.get("io") == "host":
            st["q"] = q
        else:
            st["x0"], st["out"] = _device_io(w, q)
        if kind == "closure":
            from phi_eng_b200.closure import Mlp

            st["mlp"] = Mlp.load(os.path.join(ROOT, "phi_eng_b200", "weights", "closure_mlp.npz"))
            w.set_closure(st["mlp"])
    elif kind == "batch2":
        from phi_eng_b200.batch import Batch

        scs = _batch_scenes(case, seed)
        b = Batch([_world2(case, q, None, boxes, [], g) for q, boxes, g in scs])
        _precision(b.world, case["mode"])
        q = np.concatenate([q for q, _, _ in scs])
        st.update(b=b, n=len(q))
        st["x0"], st["out"] = _device_io(b.world, q)
    elif kind == "fluid3":
        from phi_eng_b200 import _abi
        from phi_eng_b200.world3 import Box3, World3

        q, boxes = _scene3(case, seed)
        cfg, rest, mass, _, _ = _config(case)
        w = World3()
        _precision(w, case["mode"])
        for b in boxes:
            w.add_static_body(b[:3], Box3(*b[3:]))
        w.fluid.config = _ffi(cfg, rest, mass, _abi.default_config())
        w.fluid.set_cap(max(4096, len(q)))
        w.fluid.add_particles(q[:, :3])
        w.fluid.set_state(q)
        st.update(w=w, q=q)
    else:
        from phi_eng_b200.closure import Mlp

        x, t, p, norm = _pairs(case, seed)
        st.update(x=x.cuda(), t=t.cuda(), p=p, norm=norm, mlp=Mlp())
    return st


def run(st):
    case, kind, dt = st["case"], st["case"]["kind"], st["dt"]
    if kind == "fluid2" and case["io"] == "host":
        w = st["w"]
        w.fluid.set_state(st["q"])
        for _ in range(case["steps"]):
            w.step(dt)
        return w.fluid.particles
    if kind in ("fluid2", "batch2"):
        w = st["w"] if kind == "fluid2" else st["b"].world
        w.set_state_device(st["x0"].data_ptr(), st["n"])
        w.step_n(dt, case["steps"])
        w.get_state_device(st["out"].data_ptr(), st["n"])
        return st["out"]
    if kind == "closure":
        w = st["w"]
        w.set_state_device(st["x0"].data_ptr(), st["n"])
        stats = w.closure_step(dt, case["steps"])
        w.get_state_device(st["out"].data_ptr(), st["n"])
        return {"state": st["out"], "coarse": int(stats.coarse_steps)}
    if kind == "fluid3":
        st["w"].fluid.set_state(st["q"])
        st["w"].step_n(dt, case["steps"])
        return st["w"].fluid.particles
    m = st["mlp"]
    m.set(st["p"], st["norm"])
    hist = m.train(st["x"], st["t"], batch=case["batch"], iters=case["iters"], lr=1e-3, seed=0xC105E)
    return {"loss": hist, "params": m.get()[0]}


def work(case):
    """Bytes: the state in and out once (16 B a 2D particle, 24 B a 3D one), or the sampled pairs. Operations:
    per step, the pairs inside the support (about 12.6 in 2D and 33.5 in 3D, the particle itself among them) at
    what one density and one force term take, and the advance of each particle."""
    kind = case["kind"]
    if kind == "train":
        net = 2 * (16 * 64 + 64 * 64 + 64 * 2)
        return {"bytes": case["iters"] * case["batch"] * 72.0, "flops": case["iters"] * case["batch"] * 3.0 * net}
    if kind == "fluid3":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 48.0 * n, "flops": case["steps"] * n * (33.5 * (14 + 40) + 60.0)}
    n = sum(s[0] for s in _batch_shapes(case, 1)) if kind == "batch2" else case["nx"] * case["ny"]
    per = 12.6 * (11 + 32) + 50.0
    if kind == "closure":
        per += 12.6 * 30 + 2 * (16 * 64 + 64 * 64 + 64 * 2)
    sub = 2 if case.get("terms") == "all" else 1
    return {"bytes": 32.0 * n, "flops": case["steps"] * sub * n * per}


# ---------------------------------------------------------------- 64-bit values
def _f64_pairs(pos, scene, h):
    """(i, j) of every pair with |x_i - x_j| < h inside one scene, i == j among them."""
    dev, D = pos.device, pos.shape[1]
    cell = torch.floor(pos / h).long()
    cell -= cell.min(0).values - 1
    dims = (cell.max(0).values + 2).tolist()
    key = scene.clone()
    for a in range(D):
        key = key * dims[a] + cell[:, a]
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=int(math.prod(dims)) * (int(scene.max()) + 1))
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    ids = torch.arange(len(pos), device=dev)
    I, J = [], []
    for o in range(3 ** D):
        off, m = 0, o
        for a in range(D):
            off, m = off * dims[a] + (m % 3 - 1), m // 3
        k = key + off
        first, many = start[k], count[k]
        for t in range(most):
            i = ids[many > t]
            j = order[first[i] + t]
            d = pos[i] - pos[j]
            near = (d * d).sum(1) < h * h
            I.append(i[near])
            J.append(j[near])
    return torch.cat(I), torch.cat(J)


def _f64_density(pos, scene, S):
    n, h, D = len(pos), S["h"], pos.shape[1]
    i, j = _f64_pairs(pos, scene, h)
    d = pos[i] - pos[j]
    r2 = (d * d).sum(1)
    W = (4.0 / (math.pi * h ** 8) if D == 2 else 315.0 / (64.0 * math.pi * h ** 9)) * (h * h - r2) ** 3
    rho = torch.zeros(n, dtype=torch.float64, device=pos.device).index_add_(0, i, S["m"][j] * W)
    rho = rho.clamp(0.0, 3.0 * S["rho0"])
    if S["gamma"] == 1.0:
        p = (S["k"] * (rho - S["rest"])).clamp_min(0.0)
    else:
        p = (S["k"] * S["rest"] * ((rho / S["rest"]) ** S["gamma"] - 1.0)).clamp_min(0.0)
    off = i != j
    return rho, p, (i[off], j[off], d[off], r2[off], W[off])


def _f64_walls(pos, vel, S):
    for b, kind in S["bodies"]:
        D = pos.shape[1]
        rel = pos - b[:, :D]
        if kind == "circle":
            dist = rel.norm(dim=1)
            rr = b[:, D] + S["pr"]
            hit = dist < rr
            nrm = rel / dist.clamp_min(1e-300)[:, None]
            depth = rr - dist
        else:
            half = b[:, D:]
            diff = rel - torch.maximum(torch.minimum(rel, half), -half)
            dist = diff.norm(dim=1)
            outer = dist * dist > 1e-12
            pen = half - rel.abs()
            axis = pen.argmin(1) if D == 3 else torch.where(pen[:, 0] < pen[:, 1], 0, 1)
            eject = torch.nn.functional.one_hot(axis, D).to(pos.dtype)
            nrm = torch.where(outer[:, None], diff / dist.clamp_min(1e-300)[:, None], eject)
            depth = torch.where(outer, S["pr"] - dist, S["pr"] + pen.gather(1, axis[:, None])[:, 0])
            hit = ~outer | (dist < S["pr"])
        hit = hit & (depth > 0.0)
        pos = torch.where(hit[:, None], pos + nrm * depth[:, None], pos)
        vn = (vel * nrm).sum(1)
        into = hit & (vn < 0.0)
        vel = torch.where(into[:, None], (vel - nrm * vn[:, None]) * (1.0 - S["mu"]), vel)
    return pos, vel


def _f64_forces(pos, vel, rho, p, nb, S):
    i, j, d, r2, W = nb
    h, D, m = S["h"], pos.shape[1], S["m"]
    q = p / rho.clamp_min(EPS) ** 2
    r = r2.sqrt()
    c = -30.0 / (math.pi * h ** 5) if D == 2 else -45.0 / (math.pi * h ** 6)
    g = torch.where(r < EPS, 0.0, c * (h - r) ** 2 / r.clamp_min(1e-300))[:, None] * d
    term = q[i] + q[j]
    rho_bar = 0.5 * (rho[i].clamp_min(EPS) + rho[j].clamp_min(EPS))
    dv = vel[j] - vel[i]
    if S["av"] > 0.0:
        vd = -(dv * d).sum(1)
        mu = h * vd / (r2 + 0.01 * h * h)
        term = term + torch.where((vd < 0.0) & (r > EPS), -S["av"] * math.sqrt(S["k"]) * mu / rho_bar, 0.0)
    pair = -g * (m[j] * term)[:, None]
    if S["tension"] > 0.0:
        pair = pair - torch.where(r > EPS, S["tension"] * m[i] * m[j] * (1.0 - r / h) / r.clamp_min(1e-300), 0.0)[:, None] * d
    f = torch.zeros_like(pos).index_add_(0, i, pair)
    s = torch.zeros_like(pos).index_add_(0, i, dv * (m[j] / rho_bar * W)[:, None])
    return f, s, g, dv


def _f64_advance(pos, vel, acc, s, dt, S):
    vel = vel + acc * dt + s * S["visc"]
    speed = vel.norm(dim=1, keepdim=True)
    vel = torch.where(speed > S["vmax"], vel * (S["vmax"] / speed), vel)
    return _f64_walls(pos + vel * dt, vel, S)


def _f64_setup(case, n, phases, bodies, dev):
    cfg, rest, mass, dt, _ = _config(case)
    ph = torch.zeros(n, dtype=torch.long, device=dev) if phases is None else torch.from_numpy(phases).long().to(dev)
    f = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    return {"h": cfg["smoothing_length"], "m": f(mass)[ph], "rest": f(rest)[ph], "rho0": cfg["rest_density"],
            "k": cfg["stiffness"], "gamma": cfg["gamma"], "av": cfg["artificial_viscosity"],
            "tension": cfg["surface_tension"], "mu": cfg["wall_friction"], "visc": cfg["viscosity"],
            "vmax": cfg["max_velocity"], "pr": cfg["particle_radius"], "bodies": bodies, "dt": dt,
            "cfl": cfg["cfl"], "max_substeps": cfg["max_substeps"]}


def _f64_steps(q, scene, S, grav, steps):
    D = q.shape[1] // 2
    pos, vel = q[:, :D], q[:, D:]
    for _ in range(steps):
        ns = 1
        if S["cfl"] > 0.0:
            c0 = math.sqrt(S["gamma"] * S["k"] * S["rho0"])
            ns = math.ceil(S["dt"] / (S["cfl"] * S["h"] / (c0 + float(vel.norm(dim=1).max()))))
            ns = max(1, min(ns, S["max_substeps"]))
        for _ in range(ns):
            rho, p, nb = _f64_density(pos, scene, S)
            f, s, _, _ = _f64_forces(pos, vel, rho, p, nb, S)
            pos, vel = _f64_advance(pos, vel, grav + f / rho.clamp_min(EPS)[:, None], s, S["dt"] / ns, S)
    return torch.cat([pos, vel], 1)


def _f64_net(p, x, keep=False):
    W1, b1, W2, b2, W3, b3 = p
    z1 = x @ W1.T + b1
    h1 = z1 * torch.sigmoid(z1)
    z2 = h1 @ W2.T + b2
    h2 = z2 * torch.sigmoid(z2)
    y = h2 @ W3.T + b3
    return (y, z1, h1, z2, h2) if keep else y


def _f64_unpack(v):
    out, at = [], 0
    for r, c in ((64, 16), (64, 64), (2, 64)):
        out += [v[at:at + r * c].view(r, c), v[at + r * c:at + r * c + r]]
        at += r * c + r
    return out


def _f64_closure(q, S, grav, steps, dev):
    z = np.load(os.path.join(ROOT, "phi_eng_b200", "weights", "closure_mlp.npz"))
    p = _f64_unpack(torch.from_numpy(z["params"]).double().to(dev))
    norm = torch.from_numpy(z["norm"]).double().to(dev)
    scene = torch.zeros(len(q), dtype=torch.long, device=dev)
    pos, vel, h, dt = q[:, :2], q[:, 2:], S["h"], 4.0 * S["dt"]
    kr = S["k"] * S["rest"]
    for _ in range(steps):
        rho, pr, nb = _f64_density(pos, scene, S)
        f, s, g, dv = _f64_forces(pos, vel, rho, pr, nb, S)
        i, j, _, _, W = nb
        V = S["m"][j] / rho[j].clamp_min(EPS)
        zero = torch.zeros_like(rho)
        add = lambda v: zero.clone().index_add_(0, i, v)  # noqa: E731
        sw = add(V * W)
        iw = torch.where(sw > 0.0, 1.0 / sw.clamp_min(1e-300), 0.0)
        near, nx, ny = torch.full_like(rho, 3.0 * h), zero.clone(), zero.clone()
        for b, _ in S["bodies"]:
            rel = pos - b[:, :2]
            o = rel.abs() - b[:, 2:]
            out = (o > 0.0).any(1)
            oc = o.clamp_min(0.0)
            dist = torch.where(out, oc.norm(dim=1), o.max(1).values)
            sg = torch.where(rel < 0.0, -1.0, 1.0)
            inner = torch.where((o[:, :1] >= o[:, 1:]), torch.tensor([1.0, 0.0], dtype=torch.float64, device=dev),
                                torch.tensor([0.0, 1.0], dtype=torch.float64, device=dev))
            nrm = sg * torch.where(out[:, None], oc / dist.clamp_min(1e-300)[:, None], inner)
            less = dist < near
            near = torch.where(less, dist, near)
            nx, ny = torch.where(less, nrm[:, 0], nx), torch.where(less, nrm[:, 1], ny)
        x = torch.stack([
            rho / S["rest"] - 1.0, pr / kr, add(V * (dv * g).sum(1)) * dt,
            add(V * (dv[:, 0] * g[:, 1] - dv[:, 1] * g[:, 0])) * dt, add(torch.ones_like(V)) / 16.0,
            near.clamp_min(-h) / h, nx, ny, add(V * W * dv[:, 0]) * iw * dt / h, add(V * W * dv[:, 1]) * iw * dt / h,
            add(V * W * dv[:, 0] ** 2) * iw * (dt / h) ** 2, (pr - add(V * W * pr[j]) * iw) / kr,
            add(V * W * dv[:, 1] ** 2) * iw * (dt / h) ** 2, f[:, 0] / rho.clamp_min(EPS) * dt * dt / h,
            f[:, 1] / rho.clamp_min(EPS) * dt * dt / h, vel.norm(dim=1) * dt / h], 1)
        y = _f64_net(p, (x - norm[:16]) * norm[16:32]) * norm[32:]
        acc = grav + f / rho.clamp_min(EPS)[:, None] + y * (h / (dt * dt))
        pos, vel = _f64_advance(pos, vel, acc, s, dt, S)
    return torch.cat([pos, vel], 1)


def _sample(pairs, batch, seed, it):
    """The minibatch of iteration `it`: SplitMix64's finaliser of (seed, iteration, sample), scaled to the pairs."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) ^ (np.uint64(it) << np.uint64(32)) ^ np.arange(batch, dtype=np.uint64)
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
        return (((z >> np.uint64(32)) * np.uint64(pairs)) >> np.uint64(32)).astype(np.int64)


def _f64_train(case, seed, dev):
    x, t, w, norm = _pairs(case, seed)
    x, t, v = x.double().to(dev), t.double().to(dev), torch.from_numpy(w).double().to(dev)
    nm = torch.from_numpy(norm).double().to(dev)
    B, m1, m2, hist = case["batch"], torch.zeros_like(v), torch.zeros_like(v), []
    for it in range(case["iters"]):
        at = torch.from_numpy(_sample(case["pairs"], B, 0xC105E, it)).to(dev)
        xb = (x[at] - nm[:16]) * nm[16:32]
        p = _f64_unpack(v)
        y, z1, h1, z2, h2 = _f64_net(p, xb, keep=True)
        e = y - t[at] / nm[32:]
        hist.append(float((e * e).sum()) / (2 * B))
        dy = e / B
        ds = lambda z: torch.sigmoid(z) * (1.0 + z * (1.0 - torch.sigmoid(z)))  # noqa: E731
        d2 = (dy @ p[4]) * ds(z2)
        d1 = (d2 @ p[2]) * ds(z1)
        g = torch.cat([(d1.T @ xb).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0),
                       (dy.T @ h2).reshape(-1), dy.sum(0)])
        m1 = 0.9 * m1 + 0.1 * g
        m2 = 0.999 * m2 + 0.001 * g * g
        v = v - 1e-3 * (m1 / (1 - 0.9 ** (it + 1))) / ((m2 / (1 - 0.999 ** (it + 1))).sqrt() + 1e-8)
    return {"loss": np.array(hist), "params": v.cpu().numpy()}


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    kind = case["kind"]
    if kind == "train":
        return _f64_train(case, seed, dev)
    f = lambda v: torch.tensor(np.asarray(v, np.float32), device=dev).double()  # noqa: E731
    if kind == "batch2":
        scs = _batch_scenes(case, seed)
        n = [len(q) for q, _, _ in scs]
        scene = torch.repeat_interleave(torch.arange(len(scs), device=dev), torch.tensor(n, device=dev))
        boxes, q = f([b for _, b, _ in scs]), torch.from_numpy(np.concatenate([q for q, _, _ in scs])).double().to(dev)
        S = _f64_setup(case, len(q), None, [(boxes[scene, k], "box") for k in range(boxes.shape[1])], dev)
        return _f64_steps(q, scene, S, f([g for _, _, g in scs])[scene], case["steps"])
    if kind == "fluid3":
        q, boxes = _scene3(case, seed)
        ph, circles, g = None, [], (0.0, -9.81, 0.0)
    else:
        q, ph, boxes, circles, g = _scene2(case, seed)
    n = len(q)
    bodies = [(f(b)[None].expand(n, -1), "box") for b in boxes] + [(f(b)[None].expand(n, -1), "circle") for b in circles]
    S = _f64_setup(case, n, ph, bodies, dev)
    q = torch.from_numpy(q).double().to(dev)
    if kind == "closure":
        return {"state": _f64_closure(q, S, f(g)[None], case["steps"], dev), "coarse": None}
    out = _f64_steps(q, torch.zeros(n, dtype=torch.long, device=dev), S, f(g)[None], case["steps"])
    return out if kind == "fluid2" and case["io"] == "device" else out.cpu().numpy()
