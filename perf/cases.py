"""Timed workloads of the library, by what a program asks of it.

Each case is one call pattern of a user's program through the public entry
points (flip3d_gb300.gpu and the C ABI it loads):

  step      one simulation step on a state handed over and read back, the way
            a driver of its own particles calls it: on device arrays
            (via = "device"), on pinned host arrays (via = "host"), or as a
            replayed CUDA graph on the resident state (via = "graph")
  batch     one step of several independent scenes from captured graphs
  transfer  the particle-to-grid half of a step stage by stage: sort,
            density, markWater, P2G
  correct   the corrector on its own (its sort, the spring, the resample)
  solve     the pressure solve on its own, with each preconditioner
  mesh      the surface mesh of a frame, downloaded
  predict   the warm start's network on a batch of systems
  train     one training step of that network

The scenes are the two the project's scenes module and benchmark use, a pool
with a falling sphere and a dam-break column, with seeded jitter and a smooth
seeded velocity field on top, as a moving liquid has.
"""
import ctypes
import math
import os

import numpy as np
import torch

from flip3d_gb300 import gpu, scenes

DEV = "cuda"


# ------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest scene of the batched workload, replayed frame by frame:
        # launches and latency
        {"name": "step_graph_n24", "kind": "step", "n": 24, "scene": "pool", "via": "graph",
         "arith": "fast", "precond": "mg"},
        # the library's defaults, the reference's arithmetic bit for bit, near
        # the reference's own grid
        {"name": "step_ref_n48", "kind": "step", "n": 48, "scene": "pool", "via": "device",
         "arith": "ref", "precond": "ref"},
        # a host driver's frame: particles in pinned memory, in and out
        {"name": "step_host_n128", "kind": "step", "n": 128, "scene": "dam", "via": "host",
         "arith": "fast", "precond": "mg"},
        # the headline configuration, 35M particles
        {"name": "step_n256", "kind": "step", "n": 256, "scene": "pool", "via": "device",
         "arith": "fast", "precond": "mg"},
        # scenes of uneven sizes advanced together
        {"name": "batch_15", "kind": "batch", "members": 15},
        # the stages of a driver that calls them one by one
        {"name": "transfer_n160", "kind": "transfer", "n": 160, "scene": "dam", "arith": "fast"},
        # the corrector on an odd grid
        {"name": "correct_n109", "kind": "correct", "n": 109, "scene": "pool", "arith": "fast"},
        # the pressure solve by itself: the default method on a large grid and
        # the method it is compared with
        {"name": "solve_mg_n192", "kind": "solve", "n": 192, "precond": "mg"},
        {"name": "solve_mic_n96", "kind": "solve", "n": 96, "precond": "mic"},
        # one frame's mesh
        {"name": "mesh_n100", "kind": "mesh", "n": 100, "scene": "pool", "arith": "fast"},
        # the learned warm start: inference as a solve asks for it, and a
        # training step at the training batch
        {"name": "predict_n128", "kind": "predict", "n": 128, "batch": 1},
        {"name": "train_n32_b16", "kind": "train", "n": 32, "batch": 16},
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "transfer", "transfer", "correct",
                       "correct", "solve", "solve", "solve", "mesh", "predict", "train"])
    scene = rng.choice(["pool", "dam"])
    arith = rng.choice(["fast", "fast", "ref"])
    if kind == "step":
        if rng.random() < 0.2:
            return {"kind": kind, "n": _log_int(rng, 16, 64), "scene": scene, "via": "device",
                    "arith": "ref", "precond": "ref"}
        precond = rng.choice(["mg", "mg", "jacobi"])
        n = _log_int(rng, 24, 224, 4) if precond == "mg" else _log_int(rng, 21, 151)
        return {"kind": kind, "n": n, "scene": scene,
                "via": rng.choice(["device", "host", "graph"]), "arith": arith,
                "precond": precond}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(2, 24)}
    if kind in ("transfer", "correct"):
        return {"kind": kind, "n": _log_int(rng, 17, 200), "scene": scene, "arith": arith}
    if kind == "solve":
        precond = rng.choice(["mg", "mg", "jacobi", "mic"])
        n = {"mg": lambda: _log_int(rng, 16, 224, 4), "jacobi": lambda: _log_int(rng, 15, 160),
             "mic": lambda: _log_int(rng, 15, 128)}[precond]()
        return {"kind": kind, "n": n, "precond": precond}
    if kind == "mesh":
        return {"kind": kind, "n": _log_int(rng, 16, 144), "scene": scene, "arith": arith}
    if kind == "predict":
        return {"kind": kind, "n": _log_int(rng, 16, 128, 8), "batch": rng.randint(1, 3)}
    return {"kind": kind, "n": rng.choice([16, 24, 32, 40, 48]), "batch": rng.randint(2, 12)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _objects(scene, n, depth=0.25, r=0.15):
    w = 1.0 / n
    if scene == "dam":
        return [scenes.Box((w, w, w), (0.4, 0.8, 1 - w))]
    return [scenes.Box((w, w, w), (1 - w, depth, 1 - w)),
            scenes.Sphere((0.5, 0.75, 0.5), r, (0.0, -2.0, 0.0))]


def _params(case, count, seed):
    kw = {"seed": int(seed) & 0xFFFF}
    if case.get("arith") == "fast":
        kw["arith"] = gpu.ARITH_FAST
    precond = case.get("precond", "mg" if case["n"] % 4 == 0 else "jacobi")
    if precond == "ref":  # the library's defaults
        kw["rel_tol"] = 1e-4
    else:
        kw.update(solve_mode=gpu.SOLVE_FAST, rel_tol=1e-6,
                  precond={"mg": gpu.PRECOND_MG, "jacobi": gpu.PRECOND_JACOBI,
                           "mic": gpu.PRECOND_IC}[precond])
        if precond == "mic":
            kw["mic_tau"] = 0.97
    return gpu.default_params(case["n"], count, **kw)


def _ptr(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _simulation(case, seed, objects):
    """A scene of jittered particles with a smooth velocity field:
    (simulation, pos, vel, type), the state in device arrays. The jitter is
    the scenes' own kind, uniform within a share of a cell, but kept off the
    walls, so that every seed has the same particles."""
    n = case["n"]
    share = 0.42 if case.get("scene") == "dam" else 0.34
    cap = int(8 * n ** 3 * share) + 7 * n * n + 4096
    sim = gpu.Simulation(_params(case, cap, seed))
    sim.seed_scene(objects, seed=int(seed), jitter=0.0)
    sim.calibrate_max_density()
    pos = torch.empty((sim.np, 3), device=DEV)
    vel = torch.empty_like(pos)
    typ = torch.empty(sim.np, dtype=torch.uint8, device=DEV)
    torch.cuda.synchronize()
    sim._ck(sim.lib.flipgpu_get_particles(sim.h, _ptr(pos), _ptr(vel), None, _ptr(typ), 1),
            "get_particles")
    g = _gen(seed)
    fluid = (typ == scenes.FLUID).unsqueeze(1)
    moved = pos + (torch.rand(pos.shape, device=DEV, generator=g) - 0.5) * (0.6 / n)
    moved = moved.clamp(1.01 / n, 1 - 1.01 / n)
    ph = torch.rand(9, device=DEV, generator=g) * 6.2831853
    for a in range(3):
        b, c = (a + 1) % 3, (a + 2) % 3
        vel[:, a] += (0.6 * torch.sin(6.2831853 * pos[:, b] + ph[a]) *
                      torch.cos(6.2831853 * pos[:, c] + ph[3 + a]) +
                      0.2 * torch.sin(37.0 * pos[:, a] + ph[6 + a])) * fluid[:, 0]
    pos = torch.where(fluid, moved, pos).contiguous()
    return sim, pos, vel.contiguous(), typ


def _rest_pressure(n, scene):
    """The pressure the resting pool (or column) left: the warm start."""
    c = (torch.arange(n, device=DEV, dtype=torch.float32) + 0.5) / n
    top = 0.8 if scene == "dam" else 0.25
    p = (0.006 * 9.8 * (top - c).clamp(min=0)).view(1, n, 1).expand(n, n, n).contiguous()
    if scene == "dam":
        p[int(0.4 * n):] = 0
    for d in range(3):
        p.select(d, 0).zero_()
        p.select(d, n - 1).zero_()
    return p.reshape(-1)


def _system(n, g):
    """One pressure system: cell flags, levelset, divergence and a start."""
    c = (torch.arange(n, device=DEV, dtype=torch.float32) + 0.5) / n
    x, y, z = torch.meshgrid(c, c, c, indexing="ij")
    ph = torch.rand(12, device=DEV, generator=g) * 6.2831853
    wave = 0.03 * torch.sin(6.2831853 * x + ph[0]) * torch.cos(6.2831853 * z + ph[1])
    # filling of a cell in [0, 1] from the signed distance to pool and sphere
    d = torch.maximum(0.3 + wave - y,
                      0.16 - ((x - 0.5) ** 2 + (y - 0.68) ** 2 + (z - 0.5) ** 2).sqrt())
    noise = torch.randn(n, n, n, device=DEV, generator=g)
    fill = (d * n + 0.5).clamp(0, 1) * (1 + 0.05 * noise.clamp(-2, 2))
    L = 1.6 - 8.0 * fill
    A = (L < 0).to(torch.uint8)
    div = torch.zeros(n, n, n, device=DEV)
    for m in range(3):
        div += 2.0 * torch.sin(6.2831853 * (m + 1) * x + ph[2 + m]) * \
            torch.cos(6.2831853 * (m + 1) * y + ph[5 + m]) * \
            torch.sin(6.2831853 * (m + 1) * z + ph[8 + m])
    div += 0.3 * torch.randn(n, n, n, device=DEV, generator=g)
    for s in range(3):
        for e in (0, n - 1):
            A.select(s, e).fill_(scenes.WALL)
            L.select(s, e).fill_(1.0)
    fl = A == scenes.FLUID
    div = torch.where(fl, div, torch.zeros_like(div))
    p0 = torch.where(fl, 0.006 * 9.8 * (0.3 - y).clamp(min=0), torch.zeros_like(y))
    return A.reshape(-1), L.reshape(-1), div.reshape(-1), p0.reshape(-1)


def _net_inputs(case, seed):
    """Systems of the network: flags, b, x0, r0 = b - A x0 and a target x."""
    n, g = case["n"], _gen(seed)
    got = []
    for _ in range(case["batch"]):
        A, L, div, p0 = _system(n, g)
        b = -div
        diag, nb = _matrix(A, L, n, torch.float32)
        r0 = torch.where(A == 1, b - _apply(diag, nb, p0, n) * float(n * n), torch.zeros_like(b))
        s = r0.square().sum().div((A == 1).sum()).sqrt() / (n * n)
        t = torch.randn(n, n, n, device=DEV, generator=g)
        t = torch.nn.functional.avg_pool3d(t.view(1, 1, n, n, n), 5, 1, 2).view(-1)
        got.append((A, b, p0, r0, p0 + s * (0.5 * r0 / (r0.abs().max() + 1e-20) + 4.0 * t)))
    return [torch.cat(t).contiguous() for t in zip(*got)]


WEIGHTS = os.path.join(os.path.dirname(gpu.__file__), "unet_weights.bin")

BATCH_N = (24, 32, 48, 64, 96)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "transfer", "correct", "mesh"):
        n = case["n"]
        sim, pos, vel, typ = _simulation(case, seed, _objects(case["scene"], n))
        s = {"case": case, "sim": sim, "pos": pos, "vel": vel}
        if kind == "step":
            s["press"] = _rest_pressure(n, case["scene"])
            s["out"] = [torch.empty_like(pos), torch.empty_like(vel), torch.empty_like(s["press"])]
        elif kind == "transfer":
            s["out"] = [torch.empty(sim.np, device=DEV)] + \
                [torch.empty((n + 1) * n * n, device=DEV) for _ in range(3)] + \
                [torch.empty(n ** 3, device=DEV, dtype=torch.uint8), torch.empty(n ** 3, device=DEV)]
        elif kind == "correct":
            s["out"] = [torch.empty_like(pos), torch.empty_like(vel)]
        else:
            # one set of host arrays for all frames, larger than a frame's mesh
            cap = 16 * n * n
            s["out"] = {"vertices": np.zeros((cap, 3)), "normals": np.zeros((cap, 3)),
                        "faces": np.zeros((2 * cap, 3), np.int32)}
        torch.cuda.synchronize()
        if case.get("via") == "host":
            for k in ("pos", "vel"):
                s["h" + k] = s[k].cpu().pin_memory().numpy()
                s["o" + k] = torch.empty(s[k].shape).pin_memory().numpy()
        if case.get("via") == "graph":
            sim.put_state(pos.data_ptr(), vel.data_ptr(), True)
            sim._ck(sim.lib.flipgpu_set_grid(sim.h, None, None, None, None, None,
                                             _ptr(s["press"]), None, 1), "set_grid")
            sim.capture_step()
        return s
    if kind == "batch":
        rng = np.random.default_rng(int(seed))
        sims, outs = [], []
        for m in range(case["members"]):
            n = BATCH_N[m % len(BATCH_N)]
            depth, r = 0.12 + 0.03 * (m % 7), 0.08 + 0.02 * (m % 6)
            c = {"n": n, "arith": "fast", "precond": "mg", "scene": "dam"}
            sim, pos, vel, _ = _simulation(c, int(rng.integers(1 << 30)),
                                           _objects("pool", n, depth, r))
            torch.cuda.synchronize()
            sim.put_state(pos.data_ptr(), vel.data_ptr(), True)
            sim.sync()
            sims.append(sim)
            outs.append((torch.empty_like(pos), torch.empty_like(vel)))
        batch = gpu.Batch(sims)
        batch.capture()
        return {"case": case, "batch": batch, "out": outs}
    if kind == "solve":
        n = case["n"]
        sim = gpu.Simulation(_params(case, 1024, seed))
        sys_ = _system(n, _gen(seed))
        torch.cuda.synchronize()
        return {"case": case, "sim": sim, "sys": sys_, "out": torch.empty(n ** 3, device=DEV)}
    net = gpu.UNet(seed=0)
    net.load(WEIGHTS)
    sys_ = _net_inputs(case, seed)
    torch.cuda.synchronize()
    return {"case": case, "net": net, "sys": sys_, "out": torch.empty_like(sys_[1])}


# --------------------------------------------------------------------- run

def _read(sim, pos=None, vel=None, dens=None):
    sim._ck(sim.lib.flipgpu_get_particles(sim.h, _ptr(pos), _ptr(vel), _ptr(dens), None, 1),
            "get_particles")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim = state["sim"]
        pos, vel, press = state["out"]
        if case["via"] == "graph":
            sim.step_graph()
            _read(sim, pos, vel)
            return {"pos": pos, "vel": vel}
        sim._ck(sim.lib.flipgpu_set_grid(sim.h, None, None, None, None, None,
                                         _ptr(state["press"]), None, 1), "set_grid")
        if case["via"] == "host":
            sim.step_host(state["hpos"], state["hvel"], state["opos"], state["ovel"])
            pos, vel = state["opos"], state["ovel"]
        else:
            sim.put_state(state["pos"].data_ptr(), state["vel"].data_ptr(), True)
            sim.step()
            _read(sim, pos, vel)
        sim._ck(sim.lib.flipgpu_get_grid(sim.h, None, None, None, None, None, _ptr(press), None,
                                         1), "get_grid")
        return {"pos": pos, "vel": vel, "press": press}
    if kind == "batch":
        state["batch"].step()
        for sim, (pos, vel) in zip(state["batch"].sims, state["out"]):
            _read(sim, pos, vel)
        return state["out"]
    if kind == "transfer":
        sim = state["sim"]
        dens, u0, u1, u2, A, L = state["out"]
        sim.put_state(state["pos"].data_ptr(), state["vel"].data_ptr(), True)
        sim.sort()
        sim.compute_density()
        sim.mark_water()
        sim.p2g()
        _read(sim, dens=dens)
        sim._ck(sim.lib.flipgpu_get_grid(sim.h, _ptr(u0), _ptr(u1), _ptr(u2), _ptr(A), _ptr(L),
                                         None, None, 1), "get_grid")
        return {"dens": dens, "u0": u0, "u1": u1, "u2": u2, "A": A, "L": L}
    if kind == "correct":
        sim = state["sim"]
        pos, vel = state["out"]
        sim.put_state(state["pos"].data_ptr(), state["vel"].data_ptr(), True)
        sim.correct()
        _read(sim, pos, vel)
        return {"pos": pos, "vel": vel}
    if kind == "solve":
        sim = state["sim"]
        A, L, div, p0 = state["sys"]
        sim._ck(sim.lib.flipgpu_set_grid(sim.h, None, None, None, _ptr(A), _ptr(L), _ptr(p0),
                                         _ptr(div), 1), "set_grid")
        sim.solve()
        sim._ck(sim.lib.flipgpu_get_grid(sim.h, None, None, None, None, None,
                                         _ptr(state["out"]), None, 1), "get_grid")
        return {"press": state["out"]}
    if kind == "mesh":
        sim = state["sim"]
        sim.put_state(state["pos"].data_ptr(), state["vel"].data_ptr(), True)
        sim.sort()
        nv, nf = sim.mesh_counts()
        out = state["out"]
        if nv > len(out["vertices"]) or nf > len(out["faces"]):
            raise ValueError("the frame's mesh is larger than the arrays")
        sim._ck(sim.lib.flipgpu_get_mesh(sim.h, *[a.ctypes.data_as(ctypes.c_void_p)
                                                  for a in out.values()], None), "get_mesh")
        return {**out, "counts": np.array([nv, nf])}
    net = state["net"]
    n, batch = case["n"], case["batch"]
    A, b, x0, r0, x = (t.data_ptr() for t in state["sys"])
    if kind == "predict":
        net.predict(n, batch, A, b, x0, r0, state["out"].data_ptr())
        return {"delta": state["out"]}
    loss = net.train_step(n, batch, A, b, x0, r0, x, 1e-3)
    return {"loss": loss, "params": net.params()}


# -------------------------------------------------------------------- work

_UNET = [(16, 16, 0), (16, 16, 0), (16, 32, 1), (32, 32, 1), (32, 48, 2), (48, 48, 2),
         (48, 64, 3), (64, 64, 3), (112, 48, 2), (48, 48, 2), (80, 32, 1), (32, 32, 1),
         (48, 16, 0), (16, 16, 0)]


def _share(scene, depth=0.25, r=0.15):
    return 0.32 if scene == "dam" else depth + 4.19 * r ** 3


def _step_work(n, share):
    """A step's particles (8 a liquid cell): positions and velocities in and
    out, the pressure in and out; the density's, the transfer's and the
    corrector's pair terms and about ten passes of the solver's matrix."""
    p, c = 8 * n ** 3 * share, float(n ** 3)
    return {"bytes": 49.0 * p + 8 * c, "flops": p * (216 * 9 + 54 * 12 + 2 * 64 * 9) +
            c * share * 10 * 14}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        got = [_step_work(BATCH_N[m % 5], _share("pool", 0.12 + 0.03 * (m % 7),
                                                 0.08 + 0.02 * (m % 6)))
               for m in range(case["members"])]
        return {k: sum(w[k] for w in got) for k in ("bytes", "flops")}
    n = case["n"]
    c = float(n ** 3)
    if kind == "step":
        return _step_work(n, _share(case["scene"]))
    if kind in ("transfer", "correct", "mesh"):
        p = 8 * c * _share(case["scene"])
        if kind == "transfer":
            return {"bytes": 29 * p + 12 * c + 5 * c, "flops": p * (216 * 9 + 54 * 12)}
        if kind == "correct":
            return {"bytes": 49 * p, "flops": p * 2 * 64 * 9}
        faces = 9.0 * n * n
        return {"bytes": 13 * p + faces * (24 + 12), "flops": c * 60}
    if kind == "solve":
        # the system once in, the pressure once out; ten applications of the
        # seven-point matrix on the liquid are the least a solve takes
        return {"bytes": 17 * c, "flops": 0.35 * c * 10 * 14}
    cells = case["batch"] * c
    macs = sum(27.0 * ci * co * cells / 8 ** lv for ci, co, lv in _UNET)
    if kind == "predict":
        return {"bytes": 17 * cells, "flops": 2 * macs}
    return {"bytes": 17 * cells + 2 * 4 * 684817.0, "flops": 6 * macs}


# ------------------------------------------------------- values in 64 bits

def _matrix(A, L, n, dtype):
    """Diagonal and liquid-neighbour flags of the seven-point operator with
    the subcell (ghost-fluid) diagonal, h = 1."""
    A3, L3 = A.view(n, n, n), L.view(n, n, n).to(dtype)
    fl = A3 == scenes.FLUID
    diag = torch.zeros_like(L3)
    low = torch.clamp(L3, max=1e-6)
    nb = []
    for d in range(3):
        for o in (-1, 1):
            An = torch.roll(A3, o, d)
            Ln = torch.roll(L3, o, d)
            e = 0 if o == 1 else n - 1  # the rolled-in plane lies outside the grid
            An.select(d, e).fill_(scenes.WALL)
            diag += torch.where(An == scenes.WALL, torch.zeros_like(L3), torch.ones_like(L3))
            diag -= torch.where(An == 0, Ln / low, torch.zeros_like(L3))
            nb.append((o, d, fl & (An == scenes.FLUID)))
    return torch.where(fl, diag, torch.zeros_like(diag)), nb


def _apply(diag, nb, x, n):
    x3 = x.view(n, n, n)
    y = diag * x3
    for o, d, ok in nb:
        y -= torch.where(ok, torch.roll(x3, o, d), torch.zeros_like(x3))
    return y.view(-1)


def _solve64(A, L, div, x0, n):
    diag, nb = _matrix(A, L, n, torch.float64)
    fl = A == scenes.FLUID
    inv = torch.where(fl, 1.0 / diag.view(-1), torch.zeros_like(diag.view(-1)))
    b = torch.where(fl, -div.double() / float(n * n), torch.zeros_like(inv))
    x = torch.where(fl, x0.double(), torch.zeros_like(inv))
    r = b - _apply(diag, nb, x, n)
    z = inv * r
    p, rz, stop = z.clone(), torch.dot(r, z), 1e-12 * float(b.norm())
    for it in range(6000):
        q = _apply(diag, nb, p, n)
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if it % 25 == 24 and float(r.norm()) <= stop:
            break
        z = inv * r
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return torch.where(fl, x, x0.double())


class _Cells:
    """Particles of each cell as a padded table of indices."""

    def __init__(self, pos, n):
        self.n = n
        c = (pos * np.float32(n)).clamp(0, n - 1).to(torch.int64)
        self.c = c
        key = (c[:, 0] * n + c[:, 1]) * n + c[:, 2]
        order = torch.argsort(key, stable=True)
        count = torch.bincount(key, minlength=n ** 3)
        start = torch.cumsum(count, 0) - count
        self.k = int(count.max())
        self.table = torch.full((n ** 3 + 1, self.k), -1, device=DEV, dtype=torch.int32)
        rank = torch.arange(len(key), device=DEV) - start[key[order]]
        self.table[key[order], rank] = order.to(torch.int32)

    def around(self, cell):
        """For cells [m, 3]: the particles of each of the 27 cells there,
        index tables [m, k] with -1 for none, one after another."""
        n = self.n
        for o in range(27):
            q = cell + torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device=DEV)
            ok = ((q >= 0) & (q < n)).all(1)
            key = torch.where(ok, (q[:, 0] * n + q[:, 1]) * n + q[:, 2],
                              torch.full_like(q[:, 0], n ** 3))
            yield self.table[key].long()


def _chunks(ids, k):
    return torch.split(ids, max(1, (1 << 25) // max(k, 1)))


def _density64(pos, typ, n):
    """Sum of max(0, 1 - r^2/R^2), R = 2 cells, over the liquid of the 27
    cells around, over the peak of that sum on the calibration lattice."""
    def sums(p, t):
        cells = _Cells(p, n)
        p64 = p.double()
        out = torch.ones(len(p), device=DEV, dtype=torch.float64)
        for ids in _chunks(torch.nonzero(t == scenes.FLUID)[:, 0], cells.k):
            acc = torch.zeros(len(ids), device=DEV, dtype=torch.float64)
            for q in cells.around(cells.c[ids]):
                r2 = (p64[q] - p64[ids].unsqueeze(1)).square().sum(2)
                w = (1.0 - r2 / (2.0 / n) ** 2).clamp(min=0)
                acc += torch.where((q >= 0) & (t[q] == scenes.FLUID), w, torch.zeros_like(w)).sum(1)
            out[ids] = acc
        return out
    lat = torch.from_numpy(_lattice(n)).to(DEV)
    top = sums(lat, torch.full((len(lat),), scenes.FLUID, device=DEV, dtype=torch.uint8)).max()
    return torch.where(typ == scenes.FLUID, sums(pos, typ) / top,
                       torch.ones(len(pos), device=DEV, dtype=torch.float64))


def _lattice(n):
    """The 10^3 lattice of spacing half a cell that normalises densities."""
    h = np.float64(np.float32(0.5 / n))
    c = ((np.arange(10) + 0.5) * h).astype(np.float32)
    return np.stack([v.ravel() for v in np.meshgrid(c, c, c, indexing="ij")], 1).copy()


def _p2g64(pos, vel, typ, n):
    """Each face's weighted mean of the liquid's velocities, weights
    max(R^2/r^2 - 1, 0) with R = 1.4 cells and r^2 at least 1e-5, over the two
    cells along the face's axis and the three along the others."""
    fl = typ == scenes.FLUID
    p, v = pos[fl], vel[fl].double()
    cell = (p * np.float32(n)).clamp(0, n - 1).to(torch.int64)
    g = (p * np.float32(n)).double()
    R2 = float(np.float32(1.4) * np.float32(1.4))
    out = []
    for comp in range(3):
        ext = [n, n, n]
        ext[comp] = n + 1
        sw = torch.zeros(ext[0] * ext[1] * ext[2], device=DEV, dtype=torch.float64)
        sx = torch.zeros_like(sw)
        for o in range(27):
            off = [o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1]
            if off[comp] < 0:
                continue
            f = cell + torch.tensor(off, device=DEV)
            ok = torch.ones(len(f), device=DEV, dtype=torch.bool)
            r2 = torch.zeros(len(f), device=DEV, dtype=torch.float64)
            for d in range(3):
                ok &= (f[:, d] >= 0) & (f[:, d] < ext[d])
                r2 += (g[:, d] - (f[:, d].double() + (0.0 if d == comp else 0.5))).square()
            w = (R2 / r2.clamp(min=1e-5) - 1.0).clamp(min=0)
            ok &= w > 0
            key = ((f[:, 0] * ext[1] + f[:, 1]) * ext[2] + f[:, 2])[ok]
            sw.index_add_(0, key, w[ok])
            sx.index_add_(0, key, w[ok] * v[ok, comp])
        out.append(torch.where(sw > 0, sx / sw.clamp(min=1e-300), torch.zeros_like(sx)))
    return out


def _level64(pos, typ, dens, n):
    """0.2 * 8 - the densities of a cell's liquid; 1 where a wall particle is."""
    c = (pos * np.float32(n)).clamp(0, n - 1).to(torch.int64)
    key = (c[:, 0] * n + c[:, 1]) * n + c[:, 2]
    acc = torch.zeros(n ** 3, device=DEV, dtype=torch.float64)
    acc.index_add_(0, key, torch.where(typ == scenes.FLUID, dens, torch.zeros_like(dens)))
    wall = torch.zeros(n ** 3, device=DEV, dtype=torch.bool)
    wall[key[typ == scenes.WALL]] = True
    return torch.where(wall, torch.ones_like(acc), 0.2 * 8 - acc)


def _mix64(z):
    with np.errstate(over="ignore"):
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _draws(seed, comp, a, b):
    """The keyed draws of the corrector's close-pair kicks at step 0."""
    with np.errstate(over="ignore"):
        h = _mix64(np.uint64(seed) ^ np.uint64(0x9E3779B97F4A7C15))
        h = _mix64(h ^ np.uint64((2 << 56) | comp))
        h = _mix64(h + a.astype(np.uint64))
        h = _mix64(h + (b.astype(np.uint64) ^ np.uint64(0x632BE59BD9B4E019)))
    return (h >> np.uint64(33)).astype(np.int64)


def _wall_normals(pos, n):
    """Normals of the cube's wall particles: +1 at a low side, -1 at a high
    one, along every axis it lies at the side of, at unit length."""
    p, w = pos.double(), 1.0 / n
    nrm = (p <= 1.1 * w).double()
    nrm = torch.where(p >= 1.0 - 1.1 * w, -torch.ones_like(p), nrm)
    return nrm / nrm.norm(dim=1, keepdim=True).clamp(min=1e-30)


def _correct64(pos, vel, typ, n, seed):
    """Spring displacements among particles closer than half a cell, then the
    velocities resampled at the moved positions."""
    cells = _Cells(pos, n)
    re, dt = 0.5 / n, float(np.float32(0.006))
    p64, v64 = pos.double(), vel.double()
    new, out = p64.clone(), v64.clone()
    nrm = _wall_normals(pos, n)
    ids_all = torch.nonzero(typ == scenes.FLUID)[:, 0]
    for ids in _chunks(ids_all, cells.k):
        acc = torch.zeros(len(ids), 3, device=DEV, dtype=torch.float64)
        for q in cells.around(cells.c[ids]):
            d = p64[ids].unsqueeze(1) - p64[q]
            dist = d.square().sum(2).sqrt()
            ok = (q >= 0) & (q != ids.unsqueeze(1)) & (dist < re)
            far = ok & (dist > 0.1 * re)
            w = 50.0 * (1.0 - (dist / re) ** 2).clamp(min=0) / dist.clamp(min=1e-30) * re
            acc += torch.where(far.unsqueeze(2), w.unsqueeze(2) * d, torch.zeros_like(d)).sum(1)
            row, col = torch.nonzero(ok & ~far, as_tuple=True)
            if len(row):
                o = q[row, col]
                kick = torch.zeros(len(row), 3, device=DEV, dtype=torch.float64)
                for c in range(3):
                    r = _draws(seed, c, ids[row].cpu().numpy(), o.cpu().numpy()) % 101
                    kick[:, c] = torch.from_numpy(r.astype(np.float64)).to(DEV) * \
                        (0.01 * re / dt / 100.0)
                kick = torch.where((typ[o] == scenes.FLUID).unsqueeze(1), kick,
                                   0.05 * re / dt * nrm[o])
                acc.index_add_(0, row, kick)
        new[ids] = p64[ids] + dt * acc
    for ids in _chunks(ids_all, cells.k):
        t = new[ids]
        sw = torch.zeros(len(ids), device=DEV, dtype=torch.float64)
        su = torch.zeros(len(ids), 3, device=DEV, dtype=torch.float64)
        for q in cells.around((t * n).clamp(0, n - 1).to(torch.int64)):
            r2 = (t.unsqueeze(1) - p64[q]).square().sum(2)
            w = (re * re / r2.clamp(min=1e-5) - 1.0).clamp(min=0)
            w = torch.where((q >= 0) & (typ[q] == scenes.FLUID), w, torch.zeros_like(w))
            sw += w.sum(1)
            su += (w.unsqueeze(2) * v64[q]).sum(1)
        got = su / sw.clamp(min=1e-300).unsqueeze(1)
        out[ids] = torch.where((sw > 0).unsqueeze(1), got, v64[ids])
    return new, out


def _unet64(params, n, batch, A, b, x0, r0):
    """Output of the network and the target's scale, [batch, n, n, n]."""
    F = torch.nn.functional
    W, B, off = [], [], 0
    for ci, co, _ in _UNET:
        W.append(params[off:off + 27 * ci * co].view(3, 3, 3, ci, co).permute(4, 3, 0, 1, 2))
        off += 27 * ci * co
        B.append(params[off:off + co])
        off += co
    head, bias = params[off:off + 16], params[off + 16]
    fl = (A == scenes.FLUID).view(batch, n, n, n)
    cnt = fl.sum((1, 2, 3)).clamp(min=1).double()

    def scaled(a):
        a = torch.where(fl, a.double().view(batch, n, n, n), torch.zeros(1, device=DEV).double())
        s = (a.square().sum((1, 2, 3)) / cnt).sqrt()
        s = torch.where(s > 0, s, torch.ones_like(s))
        return a / s.view(-1, 1, 1, 1), s
    (r, sr), (bb, _), (xx, _) = scaled(r0), scaled(b), scaled(x0)
    X = torch.stack([fl.double(), r, bb, xx] + [torch.zeros_like(r)] * 12, 1)

    def cv(layer, t):
        return F.relu(F.conv3d(t, W[layer], B[layer], padding=1))

    def up(t):
        return F.interpolate(t, scale_factor=2, mode="nearest")
    e0 = cv(1, cv(0, X))
    e1 = cv(3, cv(2, F.avg_pool3d(e0, 2)))
    e2 = cv(5, cv(4, F.avg_pool3d(e1, 2)))
    e3 = cv(7, cv(6, F.avg_pool3d(e2, 2)))
    d2 = cv(9, cv(8, torch.cat([up(e3), e2], 1)))
    d1 = cv(11, cv(10, torch.cat([up(d2), e1], 1)))
    d0 = cv(13, cv(12, torch.cat([up(d1), e0], 1)))
    return (d0 * head.view(1, 16, 1, 1, 1)).sum(1) + bias, sr / float(n * n), fl


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "batch", "mesh"):
        return None  # a whole step's random draws, a mesh's topology
    if kind in ("transfer", "correct"):
        n = case["n"]
        sim, pos, vel, typ = _simulation(case, seed, _objects(case["scene"], n))
        sim.close()
        if kind == "correct":
            p, v = _correct64(pos, vel, typ, n, int(seed) & 0xFFFF)
            return {"pos": p, "vel": v}
        dens = _density64(pos, typ, n)
        u0, u1, u2 = _p2g64(pos, vel, typ, n)
        return {"dens": dens, "u0": u0, "u1": u1, "u2": u2, "A": None,
                "L": _level64(pos, typ, dens, n)}
    if kind == "solve":
        n = case["n"]
        A, L, div, p0 = _system(n, _gen(seed))
        return {"press": _solve64(A, L, div, p0, n)}
    n, batch = case["n"], case["batch"]
    if batch * n ** 3 > 2.2e6:
        return None
    A, b, x0, r0, x = _net_inputs(case, seed)
    params = torch.from_numpy(np.fromfile(WEIGHTS, np.float32)).to(DEV).double()
    if kind == "predict":
        with torch.no_grad():
            out, s, fl = _unet64(params, n, batch, A, b, x0, r0)
            out = out * s.view(-1, 1, 1, 1)
            return {"delta": torch.where(fl, out, torch.zeros_like(out)).reshape(-1)}
    params.requires_grad_(True)
    out, s, fl = _unet64(params, n, batch, A, b, x0, r0)
    t = (x.double() - x0.double()).view(batch, n, n, n) / s.view(-1, 1, 1, 1)
    loss = torch.where(fl, out - t, torch.zeros_like(out)).square().sum() / fl.sum()
    loss.backward()
    g = params.grad
    # Adam's first step (beta 0.9, 0.999, epsilon 1e-8)
    new = params.detach() - 1e-3 * g / (g.abs() + 1e-8)
    return {"loss": loss.detach(), "params": new}
