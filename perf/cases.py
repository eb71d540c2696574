"""The work a user of this framework has it do, as cases that can be timed.

Every case is one call sequence through the public entry points (the C ABI of
include/fsph.h and its Python classes) on inputs made from a seed.  The fluid
states stand for a flow some time after a dam broke: blocks of particles on a
disordered lattice, moving with a smooth rolling velocity plus a little noise;
the corrections that a step then makes are those of such a flow (half of them
below 0.001 h, one in ten thousand above 0.01 h) and so are its iterations.  A
simulation pass re-imposes that state through fsph_set_array (the round trip
of a host-coupled program: write positions and velocities, step, read the
results), so every pass does the same work.

Sizes are those of the repository's configurations (scenes.py, bench.py) and
tests, from the 4,096-particle single pass to the 16,777,216-particle drop.
"""
import ctypes
import math

import numpy as np
import torch

from fltk_sph_ice_gb300 import PBFBatch, abi, rxPBDSPH, rxSPH, scenes, warmstart

H = float(np.float32(0.0457))  # the kernel radius of every configuration
REST = float(np.float32(998.29))
DT = float(np.float32(0.0016))
DT_SPH = float(np.float32(1e-3))
SPH_MASS = float(np.float32(0.02))
NET = 32 * 64 + 64 + 64 * 64 + 64 + 64 * 3 + 3  # weights and biases of the warm-start network


def listed():
    return [
        # one density / scaling-factor pass on a small cloud, device in and out, nothing allocated:
        # the real-time-loop entry point, bound by latency and launches
        {"name": "lambda pass 4k", "kind": "lambda", "bx": 16, "by": 16, "bz": 16},
        # a small PBF scene (the size of the benchmark's FP64 replica), 10 fixed iterations
        {"name": "pbf step 7k", "kind": "pbf", "bx": 12, "by": 12, "bz": 24, "iters": 10, "skin": 0.1, "clamp": 1},
        # the configured WCSPH dam break: one explicit step
        {"name": "wcsph step 32k", "kind": "wcsph", "bx": 32, "by": 32, "bz": 32},
        # the same solver at a size that fills the GPU, ragged dimensions
        {"name": "wcsph step 1M", "kind": "wcsph", "bx": 101, "by": 97, "bz": 103},
        # the configured plain PBF dam break: 4 iterations, the reference's two-sided constraint
        {"name": "pbf step 262k", "kind": "pbf", "bx": 64, "by": 32, "bz": 64, "iters": 4, "skin": 0.05, "clamp": 0},
        # the benchmark size, iterating until the mean density error is 0.1 %
        {"name": "pbf step 1M to 0.1%", "kind": "pbf", "bx": 64, "by": 64, "bz": 128, "iters": 0, "skin": 0.1,
         "clamp": 1},
        # the same with the learned warm start (network inference, features, fewer iterations)
        {"name": "pbf warm step 1M to 0.1%", "kind": "pbf", "bx": 64, "by": 64, "bz": 128, "iters": 0, "skin": 0.1,
         "clamp": 1, "warm": 1},
        # the 16.8M-particle drop onto boundary particles, compensated sums
        {"name": "pbf drop 16M", "kind": "drop", "side": 256, "iters": 6, "skin": 0.05},
        # 256 independent scenes of 2,048 to 65,536 particles stepped together
        {"name": "batch of 256 scenes", "kind": "batch", "scenes": 256, "lo": 2048, "hi": 65536, "iters": 4},
        # the neighbour sets of every particle, as a program outside the solver asks for them (host CSR)
        {"name": "neighbour sets 64k", "kind": "neighbours", "bx": 40, "by": 40, "bz": 41},
        # the density field a surface mesher samples every frame
        {"name": "density lattice 262k", "kind": "lattice", "bx": 64, "by": 64, "bz": 64, "step": 0.5},
        # loss and gradient of the warm-start network over a training batch
        {"name": "network gradient 64k", "kind": "network", "rows": 65536},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, lo, hi):
    """Ragged block dimensions holding about log-uniform [lo, hi] particles: by <= bx, bz <= 2 bx."""
    n = _log(rng, lo, hi)
    a, b = rng.uniform(0.5, 1.0), rng.uniform(0.6, 2.0)
    bx = max(4, round((n / (a * b)) ** (1.0 / 3.0)))
    by = max(2, min(bx, round(a * bx)))
    return {"bx": bx, "by": by, "bz": max(2, min(2 * bx, int(n / (bx * by))))}


def draw(rng):
    kind = rng.choice(["lambda", "pbf", "pbf", "pbf", "wcsph", "wcsph", "drop", "batch", "neighbours", "lattice",
                       "network"])
    if kind == "lambda":
        return {"kind": kind, **_block(rng, 600, 60000)}
    if kind == "pbf":
        tol = rng.random() < 0.4
        c = {"kind": kind, **_block(rng, 1000, 500000), "iters": 0 if tol else rng.choice([2, 4, 7, 10]),
             "skin": rng.choice([0.05, 0.1]), "clamp": 1 if tol else rng.randint(0, 1)}
        if tol and rng.random() < 0.5:
            c["warm"] = 1
        return c
    if kind == "wcsph":
        return {"kind": kind, **_block(rng, 3000, 1000000)}
    if kind == "drop":
        return {"kind": kind, "side": round(_log(rng, 24, 200)), "iters": rng.choice([3, 6, 10]),
                "skin": rng.choice([0.05, 0.1])}
    if kind == "batch":
        lo = rng.choice([512, 2048])
        return {"kind": kind, "scenes": rng.randint(8, 256), "lo": lo, "hi": rng.choice([16384, 65536]),
                "iters": rng.choice([3, 4, 6])}
    if kind == "neighbours":
        return {"kind": kind, **_block(rng, 4000, 100000)}
    if kind == "lattice":
        return {"kind": kind, **_block(rng, 20000, 400000), "step": rng.choice([0.4, 0.5, 0.7])}
    return {"kind": kind, "rows": round(_log(rng, 1000, 200000))}


# ---------------------------------------------------------------- inputs

def _mass(h, rest):
    """The particle mass for which a cubic lattice of spacing h / 2 sums to the rest density."""
    g = np.arange(-3, 4) * (0.5 * h)
    x, y, z = np.meshgrid(g, g, g, indexing="ij")
    r2 = x * x + y * y + z * z
    w = 315.0 / (64.0 * math.pi * h ** 9) * np.where(r2 <= h * h, (h * h - r2) ** 3, 0.0)
    return float(np.float32(rest / w.sum()))


MASS = _mass(H, REST)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _lattice(dims, spacing, origin, jitter, gen):
    """(n, 4) float32 on the GPU: a lattice, x fastest, each coordinate moved by up to +-jitter."""
    nx, ny, nz = dims
    i = torch.arange(nx * ny * nz, device="cuda")
    x = torch.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1).to(torch.float32) * spacing
    x += torch.tensor(origin, dtype=torch.float32, device="cuda")
    x += (torch.rand(x.shape, generator=gen, device="cuda") * 2 - 1) * jitter
    return torch.cat([x, torch.zeros_like(x[:, :1])], 1).contiguous()


def _flow(pos, box, amp, noise, gen):
    """Velocities of one roll of the tank (tangent to its walls, divergence-free) plus noise."""
    kx, ky = math.pi / box[0], math.pi / box[1]
    v = torch.zeros_like(pos)
    x, y = pos[:, 0], pos[:, 1]
    v[:, 0] = amp * torch.sin(kx * x) * torch.cos(ky * y)
    v[:, 1] = -amp * (kx / ky) * torch.cos(kx * x) * torch.sin(ky * y)
    v[:, :3] += noise * torch.randn((pos.shape[0], 3), generator=gen, device="cuda")
    return v


def _walls(pos, box):
    """Inside the tank, a particle radius (h / 4) clear of its walls."""
    for a in range(3):
        pos[:, a].clamp_(0.26 * H, box[a] - 0.26 * H)
    return pos


def _state(case, seed):
    """positions, velocities (n, 4 float32, GPU) and the tank's sides."""
    gen = _gen(seed)
    k = case["kind"]
    if k == "drop":
        s, n = 0.5 * H, case["side"]
        L = 2.6 * n * 0.5 * H
        ob = 0.15 * L
        top = 0.5 * (L + ob)
        o = [0.5 * (L - n * s), top + s, 0.5 * (L - n * s)]
        pos = _lattice((n, n, n), s, o, 0.015 * H, gen)
        box = [L, L, L]
        return _walls(pos, box), _flow(pos, box, 2.0, 0.02, gen), box
    bx, by, bz = case["bx"], case["by"], case["bz"]
    if k == "wcsph":  # the spacing at which the configured mass has the rest density
        s = 0.59 * H
        box = [2.05 * bx * s, max(1.05 * by, 1.02 * bx) * s, 1.05 * bz * s]
        pos = _lattice((bx, by, bz), s, [0.6 * s] * 3, 0.05 * H, gen)
        return _walls(pos, box), _flow(pos, box, 1.5, 0.02, gen), box
    s = 0.5 * H
    L = 4.1 * bx * s
    box = [L, 0.25 * L, 0.5 * L]
    a = _lattice((bx, by, bz), s, [0.6 * s] * 3, 0.015 * H, gen)
    if k != "pbf":
        return _walls(a, box), _flow(a, box, 5.0, 0.02, gen), box
    b = _lattice((bx, by, bz), s, [L - (bx - 0.4) * s, 0.6 * s, 0.6 * s], 0.015 * H, gen)
    pos = torch.cat([a, b])
    return _walls(pos, box), _flow(pos, box, 5.0, 0.02, gen), box


def _params(case, n, box):
    p = scenes.pbf_params(H, [0.0] * 3, box, n, mass=MASS, rest_dens=REST)
    if case["kind"] == "wcsph":
        p.solver, p.mass, p.viscosity, p.xsph_c, p.vort_eps = abi.SOLVER_WCSPH, SPH_MASS, 3.5 / REST, 0.0, 0.0
    if case["kind"] in ("pbf", "drop"):
        p.cell_skin = case["skin"]
        p.clamp_constraint = case.get("clamp", 1)
        if case["iters"]:
            p.eta, p.min_iter, p.max_iter = 0.0, case["iters"], case["iters"]
        else:
            p.eta, p.min_iter, p.max_iter = 1e-3, 2, 400
        p.warm_start = case.get("warm", 0)
        p.compensated_density = 1 if case["kind"] == "drop" else 0
    return p


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(ctx, st):
    if st != abi.OK:
        raise abi.FsphError(st, (ctx.L.fsph_last_error(ctx.handle) or b"").decode())


class _Simulation:
    """A context with its state on the device and buffers for what a frame reads back."""

    def __init__(self, case, seed):
        self.case = case
        self.pos, self.vel, box = _state(case, seed)
        n = self.pos.shape[0]
        sph = case["kind"] == "wcsph"
        self.dt = DT_SPH if sph else DT
        self.ctx = (rxSPH if sph else rxPBDSPH)(_params(case, n, box))
        torch.cuda.synchronize()
        _ok(self.ctx, self.ctx.L.fsph_set_particles(self.ctx.handle, _ptr(self.pos), _ptr(self.vel), n, abi.DEVICE))
        if case["kind"] == "drop":
            ob = 0.15 * box[0]
            shell = scenes.box_surface([0.5 * (box[0] - ob)] * 3, ob, 0.3 * H, layers=10)
            self.ctx.SetBoundary(shell)
        self.out = {"position": torch.empty_like(self.pos), "velocity": torch.empty_like(self.vel),
                    "density": torch.empty(n, device="cuda")}
        if case.get("warm"):  # a running simulation: the network's inputs come from the step before
            self.ctx.SetWarmStartModel(warmstart.load_model()[0])
            self.ctx.Update(self.dt)

    def frame(self):
        c, L = self.ctx, self.ctx.L
        n = self.pos.shape[0]
        _ok(c, L.fsph_set_array(c.handle, abi.RX_POSITION, _ptr(self.pos), 0, n, abi.DEVICE))
        _ok(c, L.fsph_set_array(c.handle, abi.RX_VELOCITY, _ptr(self.vel), 0, n, abi.DEVICE))
        _ok(c, L.fsph_step(c.handle, self.dt, None, None))
        for which, key in ((abi.RX_POSITION, "position"), (abi.RX_VELOCITY, "velocity"), (abi.RX_DENSITY, "density")):
            _ok(c, L.fsph_get_array(c.handle, which, _ptr(self.out[key]), abi.DEVICE, None))
        return self.out


class _LambdaPass:
    def __init__(self, case, seed):
        pos, _, box = _state(case, seed)
        self.pos, n = pos, pos.shape[0]
        self.params = _params(case, n, box)
        self.L = abi.lib()
        self.out = {"density": torch.empty(n, device="cuda"), "lambda": torch.empty(n, device="cuda")}

    def call(self):
        st = self.L.fsph_pbf_eval_lambda_noalloc(
            ctypes.byref(self.params), _ptr(self.pos), self.pos.shape[0], _ptr(self.out["density"]),
            _ptr(self.out["lambda"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != abi.OK:
            raise abi.FsphError(st, "fsph_pbf_eval_lambda_noalloc")
        return self.out


def _noalloc_signature():
    L = abi.lib()
    L.fsph_pbf_eval_lambda_noalloc.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p,
                                               ctypes.c_void_p, ctypes.c_void_p]
    L.fsph_pbf_eval_lambda_noalloc.restype = ctypes.c_int


def _batch_blocks(case):
    """Block dimensions and box sides of each scene, evenly spread over the logarithm of [lo, hi]."""
    n = case["scenes"]
    out = []
    for i in range(n):
        target = case["lo"] * (case["hi"] / case["lo"]) ** (((i * 97) % n + 0.5) / n)
        a, b = 0.6 + 0.4 * ((i * 29) % n) / n, 0.6 + 0.8 * ((i * 53) % n) / n
        bx = max(3, round((target / (a * b)) ** (1.0 / 3.0)))
        dims = (bx, max(2, round(a * bx)), max(2, round(b * bx)))
        s = 0.5 * H
        out.append((dims, [1.6 * dims[0] * s, 1.5 * dims[1] * s, 1.05 * dims[2] * s]))
    return out


def _batch_state(case, seed):
    gen, ps, vs = _gen(seed), [], []
    for dims, box in _batch_blocks(case):
        x = _walls(_lattice(dims, 0.5 * H, [0.31 * H] * 3, 0.015 * H, gen), box)
        ps.append(x)
        vs.append(_flow(x, box, 1.5, 0.02, gen))
    return ps, vs


class _Batch:
    def __init__(self, case, seed):
        ps, vs = _batch_state(case, seed)
        self.pos, self.vel = torch.cat(ps), torch.cat(vs)
        boxes = [b for _, b in _batch_blocks(case)]
        par = []
        for x, box in zip(ps, boxes):
            p = scenes.pbf_params(H, [0.0] * 3, box, x.shape[0], mass=MASS, rest_dens=REST)
            p.min_iter = p.max_iter = case["iters"]
            par.append(p)
        self.b = PBFBatch(par, [x.shape[0] for x in ps], iterations=case["iters"])
        self.out = {"position": torch.empty_like(self.pos), "velocity": torch.empty_like(self.vel),
                    "density": torch.empty(self.pos.shape[0], device="cuda")}
        torch.cuda.synchronize()

    def frame(self):
        b, L = self.b, self.b._L
        b._check(L.fsph_batch_set_particles(b.handle, _ptr(self.pos), _ptr(self.vel), abi.DEVICE))
        b.step(DT)
        for which, key in ((abi.RX_POSITION, "position"), (abi.RX_VELOCITY, "velocity"), (abi.RX_DENSITY, "density")):
            b._check(L.fsph_batch_get_array(b.handle, which, _ptr(self.out[key]), abi.DEVICE))
        return self.out


class _Neighbours:
    def __init__(self, case, seed):
        pos, vel, box = _state(case, seed)
        n = pos.shape[0]
        self.ctx = rxPBDSPH(_params(case, n, box))
        torch.cuda.synchronize()
        _ok(self.ctx, self.ctx.L.fsph_set_particles(self.ctx.handle, _ptr(pos), _ptr(vel), n, abi.DEVICE))
        # a program that asks every frame keeps buffers with room for the densest frame
        self.offsets, self.indices = np.zeros(n + 1, np.int32), np.full(48 * n, -1, np.int32)
        self.total = ctypes.c_longlong(0)

    def call(self):
        host = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        _ok(self.ctx, self.ctx.L.fsph_neighbors(self.ctx.handle, host(self.offsets), host(self.indices),
                                                self.indices.size, ctypes.byref(self.total)))
        return {"offsets": self.offsets, "indices": self.indices, "total": self.total.value}


def _lattice_nodes(case, box):
    """Node counts, origin and spacing of the field over the part of the tank that the fluid fills, and a margin."""
    d = case["step"] * H
    s = 0.5 * H
    ext = [(case["bx"] + 4) * s, (case["by"] + 4) * s, (case["bz"] + 4) * s]
    return [int(e / d) for e in ext], [-0.003 * b for b in box], [d] * 3


class _Lattice:
    def __init__(self, case, seed):
        pos, vel, box = _state(case, seed)
        self.ctx = rxPBDSPH(_params(case, pos.shape[0], box))
        torch.cuda.synchronize()
        _ok(self.ctx, self.ctx.L.fsph_set_particles(self.ctx.handle, _ptr(pos), _ptr(vel), pos.shape[0], abi.DEVICE))
        n, o, d = _lattice_nodes(case, box)
        self.n, self.o, self.d = (ctypes.c_int * 3)(*n), (ctypes.c_double * 3)(*o), (ctypes.c_double * 3)(*d)
        self.field = torch.empty((n[2], n[1], n[0]), device="cuda")

    def call(self):
        _ok(self.ctx, self.ctx.L.fsph_density_grid(self.ctx.handle, self.n, self.o, self.d, _ptr(self.field),
                                                   abi.DEVICE))
        return self.field


def _rows(case, seed):
    """Standardised features, targets that depend on them, and a network's parameter blob (host float32)."""
    gen = _gen(seed)
    x = torch.randn((case["rows"], 32), generator=gen, device="cuda")
    x[:, 23:] = 0.0
    t = 0.01 * torch.tanh(x[:, 3:6] + 0.5 * x[:, 12:13] * x[:, 13:16]) \
        + 0.002 * torch.randn((case["rows"], 3), generator=gen, device="cuda")
    w = torch.randn(NET, generator=gen, device="cuda").cpu().numpy()
    scale = np.concatenate([np.full(32 * 64, math.sqrt(2 / 32)), np.full(64, 0.05), np.full(64 * 64, math.sqrt(2 / 64)),
                            np.full(64, 0.05), np.full(64 * 3, math.sqrt(1 / 64)), np.full(3, 0.05)])
    blob = np.concatenate([np.zeros(32), np.ones(32), w * scale, [0.01]]).astype(np.float32)
    return x, t, blob


class _Network:
    def __init__(self, case, seed):
        self.x, self.t, blob = _rows(case, seed)
        self.net = warmstart.WarmStartNet(blob)
        self.grad = np.zeros(abi.MLP_BLOB_SIZE, np.float32)
        self.loss = ctypes.c_float(0)
        torch.cuda.synchronize()

    def call(self):
        m = self.net
        m._check(m.L.fsph_mlp_gradient(m.h, _ptr(self.x), _ptr(self.t), self.x.shape[0],
                                       self.grad.ctypes.data_as(ctypes.c_void_p), ctypes.byref(self.loss)), "gradient")
        return {"gradient": self.grad, "loss": self.loss.value}


def prepare(case, seed):
    k = case["kind"]
    if k in ("pbf", "drop", "wcsph"):
        return _Simulation(case, seed).frame
    if k == "lambda":
        _noalloc_signature()
        return _LambdaPass(case, seed).call
    if k == "batch":
        return _Batch(case, seed).frame
    return {"neighbours": _Neighbours, "lattice": _Lattice, "network": _Network}[k](case, seed).call


def run(state):
    return state()


# ---------------------------------------------------------------- what a pass cannot do without

def work(case):
    """Bytes: each input read once, each output written once, and per pass of a step the particle fields
    that have to cross memory between passes (a pass needs its neighbours' results of the one before).
    Flops: the pair terms within the kernel radius, about 30 neighbours a particle."""
    k = case["kind"]
    if k == "network":
        return {"bytes": case["rows"] * 4.0 * 35, "flops": 6.0 * case["rows"] * NET}
    if k == "batch":
        n = float(sum(d[0] * d[1] * d[2] for d, _ in _batch_blocks(case)))
    elif k == "drop":
        n = float(case["side"] ** 3)
    else:
        n = float(case["bx"] * case["by"] * case["bz"]) * (2 if k == "pbf" else 1)
    if k == "lambda":
        return {"bytes": 24 * n, "flops": 30 * 22 * n}
    if k == "neighbours":
        return {"bytes": (16 + 4 + 30 * 4) * n, "flops": 30 * 8 * n}
    if k == "lattice":
        nodes = float(np.prod(_lattice_nodes(case, [1.0] * 3)[0]))
        return {"bytes": 16 * n + 4 * nodes, "flops": 30 * 14 * nodes}
    if k == "wcsph":
        return {"bytes": (32 + 36 + 60) * n, "flops": 30 * (10 + 30) * n}
    it = case["iters"] or (25 if case.get("warm") else 60)
    return {"bytes": (32 + 36 + 120 + 60 * it) * n, "flops": 30 * ((22 + 28) * it + 60) * n}


# ---------------------------------------------------------------- the same in 64 bits

def _pairs(x, y, radius):
    """(i, j) of every x[i], y[j] closer than radius (float64 points), i ascending."""
    lo = torch.minimum(x.min(0).values, y.min(0).values) - 1.5 * radius
    cx, cy = ((x - lo) / radius).floor().long(), ((y - lo) / radius).floor().long()
    g = torch.maximum(cx.max(0).values, cy.max(0).values) + 2
    key = (cy[:, 2] * g[1] + cy[:, 1]) * g[0] + cy[:, 0]
    key, order = key.sort()
    ii, jj = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            row = ((cx[:, 2] + dz) * g[1] + cx[:, 1] + dy) * g[0] + cx[:, 0]
            a, b = torch.searchsorted(key, row - 1), torch.searchsorted(key, row + 1, right=True)
            cnt = b - a
            i = torch.repeat_interleave(torch.arange(x.shape[0], device=x.device), cnt)
            j = order[torch.arange(i.shape[0], device=x.device) - (cnt.cumsum(0) - cnt)[i] + a[i]]
            near = (x[i] - y[j]).square().sum(1) < radius * radius
            ii.append(i[near])
            jj.append(j[near])
    i, j = torch.cat(ii), torch.cat(jj)
    i, at = i.sort()
    return i, j[at]


def _sum(i, n, v):
    return torch.zeros((n, *v.shape[1:]), dtype=v.dtype, device=v.device).index_add_(0, i, v)


AW = 315.0 / (64.0 * math.pi * H ** 9)
AG = -45.0 / (math.pi * H ** 6)
AL = 45.0 / (math.pi * H ** 6)


def _geometry(x, i, j):
    d = x[i] - x[j]
    r = d.square().sum(1).sqrt()
    q = (H * H - r * r).clamp(min=0)
    t = (H - r).clamp(min=0)
    g = torch.where(r > 0, AG * t * t / r.clamp(min=1e-12), torch.zeros_like(r))
    return d, r, q, g


def _lambda64(x, i, j, clamp, eps=100.0):
    d, r, q, g = _geometry(x, i, j)
    n = x.shape[0]
    rho = MASS * AW * _sum(i, n, q ** 3)
    gd = (g / REST)[:, None] * d
    sd = _sum(i, n, gd.square().sum(1)) + _sum(i, n, gd).square().sum(1)
    c = rho / REST - 1.0
    return rho, c, -(c.clamp(min=0) if clamp else c) / (sd + eps)


def _pbf64(pos, vel, lo, hi, iters, clamp, gravity=-9.81):
    """One PBF step in 64 bits: prediction, iterations, XSPH, vorticity confinement."""
    dt = DT
    n = pos.shape[0]
    v = vel.clone()
    v[:, 1] += dt * float(np.float32(gravity))
    x = torch.minimum(torch.maximum(pos + dt * v, lo), hi)
    i, j = _pairs(x, x, 1.3 * H)
    wq = AW * (H * H - (0.2 * H) ** 2) ** 3
    it = 0
    while True:
        rho, c, lam = _lambda64(x, i, j, clamp)
        it += 1
        d, r, q, g = _geometry(x, i, j)
        sc = -0.1 * (AW * q ** 3 / wq) ** 4 * dt * dt
        x = x + _sum(i, n, ((lam[i] + lam[j] + sc) * g / REST)[:, None] * d)
        x = torch.minimum(torch.maximum(x, lo), hi)
        err = float(c.clamp(min=0).mean())
        if it >= (iters or 400) or (not iters and it >= 2 and err <= 1e-3):
            break
    v = (x - pos) / dt
    d, r, q, g = _geometry(x, i, j)
    vij, vol = v[j] - v[i], (MASS / rho)[j]
    om = _sum(i, n, torch.linalg.cross(vij, (-g * vol)[:, None] * d))
    vn = v + 0.01 * _sum(i, n, (AW * q ** 3 * vol)[:, None] * vij)
    m = om.square().sum(1).sqrt()
    eta = _sum(i, n, (vol * (m[j] - m[i]) * g)[:, None] * d)
    en = eta.square().sum(1, keepdim=True).sqrt()
    f = 1e-4 * torch.linalg.cross(eta / en.clamp(min=1e-30), om)
    vn = torch.where(en > 1e-30, vn + dt * f, vn)
    return x, vn, rho


def _clear(box):
    """The reachable range of a tank: the walls less the particle radius h / 4, rounded as the solver's are."""
    r = float(np.float32(0.25 * H))
    t = lambda v: torch.tensor([float(np.float32(e)) for e in v], dtype=torch.float64, device="cuda")  # noqa: E731
    return t([r] * 3), t([b - r for b in box])


def _four(x):
    return torch.cat([x, torch.zeros_like(x[:, :1])], 1)


def exact(case, seed):
    k = case["kind"]
    if k in ("drop", "neighbours") or case.get("warm"):
        return None  # boundary particles, whole numbers, and a 16-bit network
    if k == "network":
        x, t, blob = _rows(case, seed)
        w = torch.from_numpy(blob.astype(np.float64)).cuda()
        parts = [p.clone().requires_grad_() for p in torch.split(w[64:-1], [2048, 64, 4096, 64, 192, 3])]
        h1 = torch.relu(x.double() @ parts[0].view(32, 64) + parts[1])
        h2 = torch.relu(h1 @ parts[2].view(64, 64) + parts[3])
        y = h2 @ parts[4].view(64, 3) + parts[5]
        loss = (y - t.double() / w[-1]).square().sum() / case["rows"]
        g = torch.autograd.grad(loss, parts)
        z = torch.zeros(64, dtype=torch.float64, device="cuda")
        return {"gradient": torch.cat([z, *g, z[:1]]), "loss": float(loss)}
    if k == "batch":
        ps, vs = _batch_state(case, seed)
        far, lo, hi = [], [], []
        for s, (x, (_, box)) in enumerate(zip(ps, _batch_blocks(case))):  # the scenes side by side, far apart
            off = torch.tensor([16.0 * s, 0.0, 0.0], dtype=torch.float64, device="cuda")
            a, b = _clear(box)
            far.append(off.expand(x.shape[0], 3))
            lo.append((a + off).expand(x.shape[0], 3))
            hi.append((b + off).expand(x.shape[0], 3))
        far = torch.cat(far)
        x, v, rho = _pbf64(torch.cat(ps)[:, :3].double() + far, torch.cat(vs)[:, :3].double(), torch.cat(lo),
                           torch.cat(hi), case["iters"], False)
        return {"position": _four(x - far), "velocity": _four(v), "density": rho}
    pos, vel, box = _state(case, seed)
    x, v = pos[:, :3].double(), vel[:, :3].double()
    if k == "lambda":
        rho, _, lam = _lambda64(x, *_pairs(x, x, 1.01 * H), False)
        return {"density": rho, "lambda": lam}
    if k == "lattice":
        n, o, d = _lattice_nodes(case, box)
        ax = [o[a] + d[a] * torch.arange(n[a], dtype=torch.float64, device="cuda") for a in range(3)]
        z, y, xx = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
        nodes = torch.stack([xx.reshape(-1), y.reshape(-1), z.reshape(-1)], 1)
        inside = torch.ones(nodes.shape[0], dtype=torch.bool, device="cuda")
        for a in range(3):
            inside &= (nodes[:, a] >= -0.005 * box[a]) & (nodes[:, a] <= 1.005 * box[a])
        i, j = _pairs(nodes, x, H)
        w = MASS * AW * (H * H - (nodes[i] - x[j]).square().sum(1)).clamp(min=0) ** 3
        return (_sum(i, nodes.shape[0], w) * inside).reshape(n[2], n[1], n[0])
    lo, hi = _clear(box)
    if k == "wcsph":
        n = x.shape[0]
        i, j = _pairs(x, x, 1.01 * H)
        d, r, q, g = _geometry(x, i, j)
        rho = SPH_MASS * AW * _sum(i, n, q ** 3)
        p = 3.0 * (rho - REST)
        f = -SPH_MASS * _sum(i, n, ((p / rho ** 2)[i] + (p / rho ** 2)[j])[:, None] * g[:, None] * d)
        lap = torch.where(r > 0, AL * (H - r).clamp(min=0), torch.zeros_like(r))
        mu = float(np.float32(3.5 / REST))
        f += mu * SPH_MASS * _sum(i, n, (lap / rho[j])[:, None] * (v[j] - v[i]))
        f[:, 1] += float(np.float32(-9.81))
        v = v + DT_SPH * f
        x = torch.minimum(torch.maximum(x + DT_SPH * v, lo), hi)
        return {"position": _four(x), "velocity": _four(v), "density": rho}
    x, v, rho = _pbf64(x, v, lo, hi, case["iters"], bool(case["clamp"]))
    return {"position": _four(x), "velocity": _four(v), "density": rho}
