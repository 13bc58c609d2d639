"""Performance cases: what a program that uses this framework has it do, through its public
entry points, over the range of sizes and options it serves.

A case is a dict of plain values. ``kind`` names the pass:

  frame  one scene: upload a host state (lsp_write_state), take ``steps`` time steps
         (lsp_step), read back what the program looks at: positions and velocities
         (``read`` = "xv", lsp_read_particles) or the whole particle state (``read`` =
         "state", lsp_read_state). ``warm`` starts the PCISPH loop from the network's guess.
  batch  many independent scenes stepped together (lsp_batch_*), the same way.
  train  the online retraining of the warm-start network on a recorded step
         (lsp_mlp_set_weights, lsp_mlp_train, lsp_mlp_get_weights).

Every pass starts by uploading the case's state, so each pass does the same steps again. The
states are fluid in motion, not a lattice at rest: a jittered block with a smooth velocity
field, whose PCISPH loops need more than their minimum of iterations. Host buffers are pinned
and kept, as a program that steps a simulation keeps them.

``exact`` restates the reference's step in float64 torch (the tables keep the reference's 1000
divisions: they are part of what the method computes).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

SPH, PCISPH = "sph", "pcisph"


def _frame(name, solver, nx, ny, nz, spacing, steps, read="xv", factor=3.2, **kw):
    c = dict(name=name, kind="frame", solver=solver, nx=nx, ny=ny, nz=nz, spacing=spacing, steps=steps, read=read,
             factor=factor, dt_scale=0.05, jitter=0.05, speed=0.5, viscosity=0.1, eta=0.01, min_it=3, max_it=50,
             stiffness=3.0, obstacles=False, warm=False)
    c.update(kw)
    return c


def listed():
    return [
        # The smallest interactive scene: one step per call, where launches and latency count.
        _frame("pcisph_1k2", PCISPH, 10, 12, 10, 0.02, 1, obstacles=True),
        # The plain SPH dam break (12,000 particles) between two rendered frames.
        _frame("sph_12k", SPH, 20, 30, 20, 0.02, 4),
        # The reference's own defaults (h = 2.688 r, viscosity 3.5, at most 4 iterations, 10 %)
        # on an odd cube.
        _frame("pcisph_defaults_30k", PCISPH, 31, 31, 31, 0.0272, 4, factor=2.688, viscosity=3.5, eta=0.1, min_it=1,
               max_it=4),
        # A mid-size PCISPH dam break between two rendered frames.
        _frame("pcisph_102k", PCISPH, 40, 64, 40, 0.01, 4),
        # Plain SPH on a larger odd cube.
        _frame("sph_250k", SPH, 63, 63, 63, 0.008, 4),
        # The PCISPH dam break (417,792 particles) as a drop-in that owns the state on the host:
        # everything goes in and comes back each step.
        _frame("pcisph_418k_roundtrip", PCISPH, 64, 102, 64, 0.00625, 1, read="state"),
        # The largest single scene: the wave breaker's block (991,440 particles) with obstacles.
        _frame("pcisph_991k", PCISPH, 108, 68, 135, 0.00735, 4, obstacles=True),
        # A few small scenes stepped together.
        dict(name="batch_16_small", kind="batch", scenes=16, nmin=400, nmax=4000, steps=4),
        # The 64-scene batch, 2,000 to 64,000 particles each.
        dict(name="batch_64", kind="batch", scenes=64, nmin=2000, nmax=64000, steps=2),
        # Steps that start from the learned guess.
        _frame("warm_115k", PCISPH, 53, 33, 66, 0.015, 2, obstacles=True, warm=True),
        # Online retraining of the warm-start network on one recorded step of that scene.
        dict(name="train_115k", kind="train", nx=53, ny=33, nz=66, spacing=0.015, iterations=8, batch=65536),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _counts(rng, n):
    """Odd and even block counts of about n points, sides within a factor of about two."""
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    e = n ** (1.0 / 3.0)
    return [max(4, int(e * f)) for f in (a, b, 1.0 / (a * b))]


def draw(rng):
    kind = rng.choices(["frame", "batch", "warm", "train"], [10, 3, 2, 1])[0]
    if kind == "batch":
        scenes = rng.randint(3, 48)
        nmin = int(_log(rng, 300, 4000))
        return dict(kind="batch", scenes=scenes, nmin=nmin, nmax=nmin * rng.randint(2, 8), steps=rng.randint(1, 4))
    if kind == "train":
        nx, ny, nz = _counts(rng, _log(rng, 3000, 200000))
        return dict(kind="train", nx=nx, ny=ny, nz=nz, spacing=0.015, iterations=rng.randint(1, 12),
                    batch=int(_log(rng, 1000, 65536)))
    if kind == "warm":
        nx, ny, nz = _counts(rng, _log(rng, 2000, 300000))
        c = _frame(None, PCISPH, nx, ny, nz, round(_log(rng, 0.008, 0.03), 5), rng.randint(1, 3),
                   obstacles=rng.random() < 0.5, warm=True)
    else:
        n = _log(rng, 700, 700000)
        nx, ny, nz = _counts(rng, n)
        solver = rng.choice([SPH, PCISPH, PCISPH])
        c = _frame(None, solver, nx, ny, nz, round(_log(rng, 0.006, 0.03), 5), rng.randint(1, 4),
                   read=rng.choice(["xv", "xv", "state"]), factor=rng.choice([3.2, 3.2, 2.688, 3.0]),
                   obstacles=rng.random() < 0.4, viscosity=rng.choice([0.1, 1.0]))
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs

def _block(nx, ny, nz, s, jitter, speed, rng):
    """Positions and velocities of a block of fluid in motion (float32 [n, 3], x fastest): a
    jittered lattice a little off the walls, moving in a smooth field with some noise."""
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    x = np.stack([i.ravel(), j.ravel(), k.ravel()], axis=1).astype(np.float64)
    # A divergence-free roll in x and y that does not cross the walls; its sense and strength
    # come from the seed.
    ax, ay = (math.pi * (x[:, a] + 0.5) / n for a, n in ((0, nx), (1, ny)))
    a = speed * rng.uniform(0.7, 1.0) * rng.choice([-1.0, 1.0])
    v = np.stack([a * np.sin(ax) * np.cos(ay), -a * ny / nx * np.cos(ax) * np.sin(ay), np.zeros_like(ax)], axis=1)
    v += speed * rng.uniform(-0.03, 0.03, x.shape)
    x = (x + 0.75 + rng.uniform(-jitter, jitter, x.shape)) * s
    return x.astype(np.float32), v.astype(np.float32)


def _box(nx, ny, nz, s):
    """Walls of the tank: free space beside and above the block."""
    return tuple(float(np.float32(e * s)) for e in (1.6 * nx + 3.0, 1.4 * ny + 3.0, nz + 1.5))


def _scene(c, rng):
    """Everything one scene is made of: parameters, walls and obstacles, positions, velocities."""
    s = c["spacing"]
    x, v = _block(c["nx"], c["ny"], c["nz"], s, c["jitter"], c["speed"], rng)
    ext = _box(c["nx"], c["ny"], c["nz"], s)
    half = tuple(float(np.float32(0.5 * e)) for e in ext)
    cols = [("box", half, half, True)]
    if c["obstacles"]:
        # Resting on the floor beyond the block, where the fluid runs into them.
        e = float(np.float32(0.06 * min(ext)))
        cx = float(np.float32((c["nx"] + 0.75) * s + 1.6 * e))
        cols.append(("box", (cx, e, half[2]), (e, e, e), False))
        cols.append(("sphere", (cx, e, float(np.float32(0.2 * ext[2]))), e, False))
    prm = dict(particle_radius=s / 1.6, kernel_radius_factor=c["factor"], rest_density=1000.0, viscosity=c["viscosity"],
               stiffness=c["stiffness"], negative_pressure_factor=0.0, surface_tension=0.0728,
               surface_tension_threshold=7.065, restitution=0.5, friction=1.0, gravity=(0.0, -9.81, 0.0))
    if c["solver"] == PCISPH:
        prm.update(pci_eta=c["eta"], pci_min_iterations=c["min_it"], pci_max_iterations=c["max_it"])
    return prm, cols, ((0.0, 0.0, 0.0), ext), x, v, c["dt_scale"] * s


def _batch_scenes(c, rng):
    """(case of one scene, its parts) for a batch: PCISPH blocks of log-uniform sizes, which follow
    from the case (the seed makes the particles); one time step, that of the finest spacing."""
    shape = np.random.Generator(np.random.PCG64([c["scenes"], c["nmin"], c["nmax"]]))
    out = []
    for _ in range(c["scenes"]):
        n = math.exp(shape.uniform(math.log(c["nmin"]), math.log(c["nmax"])))
        a, b = shape.uniform(0.8, 1.25, 2)
        e = n ** (1.0 / 3.0)
        nx, ny, nz = (max(3, int(e * f)) for f in (a, b, 1.0 / (a * b)))
        out.append(_frame(None, PCISPH, nx, ny, nz, float(shape.uniform(0.01, 0.02)), c["steps"]))
    dt = 0.05 * min(f["spacing"] for f in out)
    return [(f, _scene(f, rng)[:5]) for f in out], dt


def _pinned(shape, dtype):
    t = torch.empty(shape, dtype=dtype, pin_memory=torch.cuda.is_available())
    return t.numpy()


def _state_arrays(x, v):
    """Host state of moving fluid: half-step velocities equal to v, no particle on its first step."""
    n = x.shape[0]
    arrs = [_pinned((n, 3), torch.float32) for _ in range(4)] + [_pinned((n,), torch.int32)]
    for a, src in zip(arrs, (x, v, v, v, 0)):
        a[...] = src
    return arrs


def _guess_weights():
    """A warm-start network that gives 0.6 f0 + 0.3 f1 for positive values (features: predicted
    density error, previous pressure): silu(z) - silu(-z) = z passes a value through a layer."""
    w1 = np.zeros((8, 32), np.float32)
    w2 = np.zeros((32, 32), np.float32)
    w3 = np.zeros((32,), np.float32)
    w1[0, 0], w1[1, 0] = 0.6, 0.3
    w1[0, 1], w1[1, 1] = -0.6, -0.3
    w2[0, 0], w2[1, 0] = 4.0, -4.0
    w3[0] = 0.25
    z = np.zeros(32, np.float32)
    return np.concatenate([w1.ravel(), z, w2.ravel(), z, w3, np.zeros(1, np.float32)])


def _solver(solver, prm, cols, dom, x, v):
    from liquidsimulation_b200 import abi, solver as S
    cls = S.PCISPHSolver if solver == PCISPH else S.SPHSolver
    s = cls(abi.default_params(**prm))
    s.set_domain(*dom)
    s.add_particles(x, v)
    for kind, center, size, boundary in cols:
        if kind == "box":
            s.add_static_collision_box(center, size, boundary)
        else:
            s.add_static_collision_sphere(center, size, boundary)
    return s


def prepare(case, seed):
    from liquidsimulation_b200 import abi, solver as S
    rng = np.random.Generator(np.random.PCG64([int(seed), 11]))
    lib = abi.load_library()
    if case["kind"] == "batch":
        scenes, dt = _batch_scenes(case, rng)
        b = S.SceneBatch()
        for f, (prm, cols, dom, x, v) in scenes:
            k = b.add_scene(abi.default_params(solver=abi.LSP_SOLVER_PCISPH, **prm), x, v, dom)
            for _, center, size, boundary in cols:
                b.add_box(k, center, size, boundary)
        x = np.concatenate([p[3] for _, p in scenes])
        v = np.concatenate([p[4] for _, p in scenes])
        host = _state_arrays(x, v)
        b.update(dt)                      # a running program: buffers and the step's graph exist
        b.update(dt)
        return dict(case=case, lib=lib, batch=b, dt=dt, host=host, out=_state_arrays(x, v), n=x.shape[0])
    if case["kind"] == "train":
        c = _frame(None, PCISPH, case["nx"], case["ny"], case["nz"], case["spacing"], 1)
        prm, cols, dom, x, v, dt = _scene(c, rng)
        s = _solver(PCISPH, prm, cols, dom, x, v)
        s.mlp_set_loss_asymmetry(4.0)
        s.mlp_record(True)
        for _ in range(4):                # the recorded step has a pressure history
            s.update(dt)
        w = rng.uniform(-0.3, 0.3, abi.MLP_PARAMS).astype(np.float32)
        return dict(case=case, solver=s, weights=w, seed=int(seed) % 1000)
    prm, cols, dom, x, v, dt = _scene(case, rng)
    s = _solver(case["solver"], prm, cols, dom, x, v)
    if case["warm"]:
        s.mlp_set_weights(_guess_weights())
        s.set_warm_start(abi.LSP_WARM_MLP)
    host = _state_arrays(x, v)
    s.update(dt)                          # a running program: its buffers exist
    n = x.shape[0]
    out = _state_arrays(x, v) if case["read"] == "state" else [_pinned((n, 3), torch.float32) for _ in range(2)]
    return dict(case=case, lib=lib, solver=s, dt=dt, host=host, out=out, n=n)


# ---------------------------------------------------------------- the pass

_F, _I = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int32)


def _ptrs(arrs):
    return [a.ctypes.data_as(_I if a.dtype == np.int32 else _F) for a in arrs]


def run(state):
    from liquidsimulation_b200 import abi
    case = state["case"]
    if case["kind"] == "train":
        s = state["solver"]
        s.mlp_set_weights(state["weights"])
        loss = s.mlp_train(iterations=case["iterations"], batch=case["batch"], lr=2e-3, seed=state["seed"])
        return dict(loss=loss, weights=s.mlp_get_weights())
    lib, n, dt = state["lib"], state["n"], state["dt"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.write_state(*state["host"])
        its = []
        for _ in range(case["steps"]):
            its.append([st.iterations for st in b.update(dt)])
        abi.check(lib, lib.lsp_batch_read_state(b._h, *_ptrs(state["out"]), n))
        its = np.array(its, np.int32)
    else:
        s = state["solver"]
        s.write_state(*state["host"])
        its = np.array([s.update(dt).iterations for _ in range(case["steps"])], np.int32)
        read = lib.lsp_read_state if case["read"] == "state" else lib.lsp_read_particles
        abi.check(lib, read(s._h, *_ptrs(state["out"]), n))
    names = ("x", "v", "half", "old", "first")
    return dict(zip(names, state["out"]), iterations=its)


# ---------------------------------------------------------------- the work of one pass

def _pairs(factor):
    return 4.18879 * (factor / 1.6) ** 3   # neighbours per particle of a lattice of spacing 1.6 r


def _step_flops(solver, factor, min_it):
    """Arithmetic of one particle's step: per pair the distance test and density (12), the
    surface tension and viscosity terms (38), and the pressure: per iteration a density (11) and
    a force (24), at least min_it of them; SPH one force (27)."""
    per_pair = 12 + 38 + (min_it * 35 if solver == PCISPH else 27)
    return _pairs(factor) * per_pair + 60.0


def work(case):
    if case["kind"] == "train":
        # Forward, data and weight gradients of the 8-32-32-1 network: 3 x 2 x 1312 per row; the
        # rows' features and targets read once per iteration, weights and moments updated.
        rows = min(case["batch"], case["nx"] * case["ny"] * case["nz"]) * case["iterations"]
        return dict(bytes=rows * 36.0 + case["iterations"] * 1377 * 24.0, flops=rows * 6.0 * 1312)
    if case["kind"] == "batch":
        n = case["scenes"] * (case["nmax"] - case["nmin"]) / math.log(max(case["nmax"] / case["nmin"], 1.001))
        return dict(bytes=n * 104.0, flops=n * case["steps"] * _step_flops(PCISPH, 3.2, 3))
    n = case["nx"] * case["ny"] * case["nz"]
    out = 52.0 if case["read"] == "state" else 24.0
    return dict(bytes=n * (52.0 + out),
                flops=n * case["steps"] * _step_flops(case["solver"], case["factor"], case["min_it"]))


# ---------------------------------------------------------------- float64 restatement

class _Exact:
    """The reference's step in float64 torch."""

    def __init__(self, prm, cols, solver, dt, x, v):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        f = np.float32
        self.p, self.cols, self.solver = prm, cols, solver
        self.dt = float(f(dt))
        self.r, self.rho0 = float(f(prm["particle_radius"])), float(f(prm["rest_density"]))
        self.mu, self.k = float(f(prm["viscosity"])), float(f(prm["stiffness"]))
        self.sig, self.thr = float(f(prm["surface_tension"])), float(f(prm["surface_tension_threshold"]))
        self.e = float(f(prm["restitution"]))
        self.h = float(f(prm["kernel_radius_factor"])) * self.r
        self.step = self.h / 1000.0
        d = np.arange(1001) * self.step
        h2 = self.h ** 2
        t = h2 - d * d
        p9, p6 = math.pi * self.h ** 9, math.pi * self.h ** 6
        tab = dict(w=315.0 / (64.0 * p9) * t ** 3, dw=-945.0 / (32.0 * p9) * t ** 2,
                   d2w=-945.0 / (32.0 * p9) * t * (3.0 * h2 - 7.0 * d * d), sdw=-45.0 / p6 * (self.h - d) ** 2,
                   vd2w=45.0 / p6 * (self.h - d))
        self.tab = {k: torch.tensor(np.append(a, 0.0), device=self.dev) for k, a in tab.items()}
        # The lattice sums behind mass and delta fall exactly on table slots: their slots are
        # those of the float32 quotients, which define them.
        s32 = f(1.6) * f(prm["particle_radius"])
        h32 = f(prm["kernel_radius_factor"]) * f(prm["particle_radius"])
        step32 = h32 / f(1000)
        g = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(f) * s32
        d32 = np.sqrt((g[:, 0] * g[:, 0] + g[:, 1] * g[:, 1]) + g[:, 2] * g[:, 2])
        slot = np.where(d32 >= h32, 1001, np.minimum((d32 / step32).astype(np.int64), 1001))
        self.mass = self.rho0 / float(np.append(tab["w"], 0.0)[slot].sum())
        gd, ok = g.astype(np.float64), d32 > 0
        grad = gd[ok] / np.linalg.norm(gd[ok], axis=1)[:, None] * np.append(tab["sdw"], 0.0)[slot[ok]][:, None]
        denom = -(grad.sum(0) ** 2).sum() - (grad ** 2).sum()
        beta = 2.0 * (self.dt * self.mass / self.rho0) ** 2
        self.delta = -1.0 / (beta * denom)
        self.g = torch.tensor([0.0, float(f(-9.81)), 0.0], dtype=torch.float64, device=self.dev)
        self.x = torch.tensor(x, device=self.dev).double()
        self.v = torch.tensor(v, device=self.dev).double()
        self.half, self.old = self.v.clone(), self.v.clone()
        self.eta = float(f(prm["pci_eta"])) if solver == PCISPH else 0.0

    def look(self, name, d):
        k = torch.where(d >= self.h, torch.full_like(d, 1001.0), torch.div(d, self.step)).clamp_(0, 1001).long()
        return self.tab[name][k]

    def neighbours(self):
        """Pairs (i, j) with |x_i - x_j| <= h, i = j included, from a sorted cell grid."""
        x, h = self.x, self.h
        c = torch.floor(x / h).long()
        lo = c.min(0).values - 1
        dims = (c.max(0).values - lo + 2).tolist()
        c = c - lo
        key = (c[:, 0] * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
        order = torch.argsort(key)
        skey = key[order]
        I, J = [], []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                row = key + (dx * dims[1] + dy) * dims[2]
                beg, end = torch.searchsorted(skey, row - 1), torch.searchsorted(skey, row + 1, right=True)
                cnt = end - beg
                i = torch.repeat_interleave(torch.arange(x.shape[0], device=self.dev), cnt)
                first = torch.cumsum(cnt, 0) - cnt
                j = order[torch.arange(i.shape[0], device=self.dev) - first[i] + beg[i]]
                keep = ((x[i] - x[j]) ** 2).sum(1) <= h * h
                I.append(i[keep].int())
                J.append(j[keep].int())
        return torch.cat(I), torch.cat(J)

    def sums(self, f, width):
        """Sum over j of f(i, j) (rows of `width`) for every particle, in chunks of pairs."""
        out = torch.zeros((self.x.shape[0], width), dtype=torch.float64, device=self.dev)
        for a in range(0, self.i.shape[0], 8_000_000):
            i, j = self.i[a:a + 8_000_000].long(), self.j[a:a + 8_000_000].long()
            out.index_add_(0, i, f(i, j))
        return out

    def collide(self, x, v):
        r = self.r
        for kind, center, size, boundary in self.cols:
            c = torch.tensor(center, dtype=torch.float64, device=self.dev)
            n, point = torch.zeros_like(x), x.clone()
            if kind == "box":
                e = torch.tensor(size, dtype=torch.float64, device=self.dev)
                dist = (c - x).abs()
                if boundary:
                    out = dist - e + r > 0
                    n = torch.where(out, torch.where(x - c <= 0, 1.0, -1.0).double(), n)
                    point = torch.where(out, c - n * (e - r), x)
                    hit = out.any(1)
                    n = n / n.norm(dim=1, keepdim=True).clamp_min(1e-300)
                else:
                    pen = e - dist + r
                    hit = (pen > 0).all(1)
                    a = torch.nn.functional.one_hot(pen.argmin(1), 3).bool()
                    n = torch.where(a, torch.where(x - c >= 0, 1.0, -1.0).double(), n)
                    point = torch.where(a, c + n * (e + r), x)
            else:
                n = x - c
                hit = (size + r) - n.norm(dim=1) > 0
                point = c + n * (size + r)
                n = n / n.norm(dim=1, keepdim=True).clamp_min(1e-300)
            sep = (v * n).sum(1, keepdim=True)
            vn = n * sep
            bounced = vn * -self.e + (v - vn)
            v = torch.where(hit[:, None] & (sep < 0), bounced, v)
            x = torch.where(hit[:, None], point, x)
        return x, v

    def run_step(self, min_it, max_it):
        x, v, dt, m = self.x, self.v, self.dt, self.mass
        self.i, self.j = self.neighbours()
        dist = lambda y, i, j: (y[i] - y[j]).norm(dim=1)  # noqa: E731
        rho = m * self.sums(lambda i, j: self.look("w", dist(x, i, j))[:, None], 1)[:, 0]

        def nonpressure(i, j):
            d, w = dist(x, i, j), 1.0 / rho[j]
            return torch.cat([(x[i] - x[j]) * (self.look("dw", d) * w)[:, None], (self.look("d2w", d) * w)[:, None],
                              (v[j] - v[i]) * (self.look("vd2w", d) * w)[:, None]], 1)

        s = self.sums(nonpressure, 7)
        normal = s[:, :3] * m
        ln = normal.norm(dim=1, keepdim=True)
        F = self.g * rho[:, None] + s[:, 4:] * (self.mu * m)
        F = F + torch.where(ln > self.thr, normal / ln.clamp_min(1e-300) * (-self.sig * s[:, 3:4] * m), 0.0 * normal)
        R = rho[:, None]

        def pressure(y, a):
            def f(i, j):
                d = dist(y, i, j)
                w = torch.where(i == j, 0.0 * d, self.look("sdw", d) * (a[i] + a[j]) / d.clamp_min(1e-300))
                return (y[i] - y[j]) * w[:, None]
            return self.sums(f, 3) * -(m * R)

        if self.solver == SPH:
            p = self.k * (rho - self.rho0)
            Fp = pressure(x, p.clamp_min(0.0) / rho ** 2)
        else:
            Fp, p = torch.zeros_like(F), torch.zeros_like(rho)
            for k in range(max_it):
                acc = (F + Fp) / R
                ph = self.half + acc * dt
                px, ph = self.collide(x + ph * dt, ph)
                pd = m * self.sums(lambda i, j: self.look("w", dist(px, i, j))[:, None], 1)[:, 0]
                er = (pd - self.rho0).clamp_min(0.0)
                p = p + self.delta * er
                Fp = pressure(px, p / pd ** 2)
                if float(er.max()) / self.rho0 < self.eta and k + 1 >= min_it:
                    break
        acc = (F + Fp) / R
        self.old = self.half
        half = self.half + acc * dt
        self.x, self.half = self.collide(x + half * dt, half)
        self.v = (self.old + self.half) / 2.0


def _exact_frame(c, parts, dt):
    prm, cols, _, x, v = parts
    e = _Exact(prm, cols, c["solver"], dt, x, v)
    for _ in range(c["steps"]):
        e.run_step(c["min_it"], c["max_it"])
    return [t.cpu().numpy() for t in (e.x, e.v, e.half, e.old)]


def exact(case, seed):
    """Positions and velocities in 64 bits. None for the iteration counts and flags, for the
    network (BF16 products and Adam's normalised steps have no 64-bit value) and for steps
    that start from its guess."""
    rng = np.random.Generator(np.random.PCG64([int(seed), 11]))
    if case["kind"] == "train" or (case["kind"] == "frame" and case["warm"]):
        return None
    if case["kind"] == "batch":
        scenes, dt = _batch_scenes(case, rng)
        got = [np.concatenate(a) for a in zip(*[_exact_frame(f, p, dt) for f, p in scenes])]
    else:
        parts = _scene(case, rng)
        got = _exact_frame(case, parts[:5], parts[5])
        if case["read"] == "xv":
            got = got[:2]
    return dict(zip(("x", "v", "half", "old"), got))
