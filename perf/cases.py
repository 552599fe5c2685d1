"""The work that users of this framework have it do, as cases that can be timed
and checked: one pass of each public path, over the range of sizes it serves.

Kinds of case
  dropin     one time step of the drop-in kernels (temperature, active lists,
             phase update) on dense device arrays, as the reference's drivers
             call them
  steps      a run segment of CompactSolver: start state restored, `steps`
             steps, the dense field written on the device
  job        a whole job: CompactSolver built from a pinned host field, stepped,
             the dense field written to pinned host memory
  batch      a segment of a BatchedBicrystals run, then every instance's field
  metrics    the observables of a state: metrics() and interface_positions()
  train      one optimiser step of the surrogate (loss, gradients, Adam)
  forward    surrogate outputs for a block of candidates
"""

from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multiphasefield-solidification-v2_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

DEVICE = "cuda:0"
UPDATE_LAUNCH = ((1, 1, 1), (4, 4, 4))  # launch geometry of the reference's drivers
MODELS = {"full": (1, 1), "no_torque": (1, 0), "isotropic": (0, 0)}  # anisotropy, torque


def listed():
    return [
        # drop-in kernels: the smallest plain-method run (8 grains, 32^3), launch latency
        {"name": "dropin-32", "kind": "dropin", "nx": 32, "ny": 32, "nz": 32, "grains": 8, "dtype": "float32",
         "checked": True, "model": "full"},
        # drop-in kernels in float64 on an odd box, plain update and unchecked lists
        {"name": "dropin-odd-f64", "kind": "dropin", "nx": 101, "ny": 90, "nz": 77, "grains": 16, "dtype": "float64",
         "checked": False, "model": "full"},
        # drop-in kernels at the headline size (256^3, 64 grains): the reference's driver loop
        {"name": "dropin-256", "kind": "dropin", "nx": 256, "ny": 256, "nz": 256, "grains": 64, "dtype": "float32",
         "checked": True, "model": "full"},
        # compact stepper on the smallest box, eager launches with the default overflow check
        {"name": "steps-32", "kind": "steps", "nx": 32, "ny": 32, "nz": 32, "grains": 8, "slots": 8, "steps": 20,
         "graph": False, "model": "full"},
        # compact stepper, isotropic model, ragged box, the widest slot template
        {"name": "steps-odd-isotropic", "kind": "steps", "nx": 150, "ny": 117, "nz": 90, "grains": 32, "slots": 16,
         "steps": 10, "graph": False, "model": "isotropic"},
        # compact stepper at the headline size, its steps captured in one graph
        {"name": "steps-256", "kind": "steps", "nx": 256, "ny": 256, "nz": 256, "grains": 64, "slots": 8, "steps": 10,
         "graph": True, "model": "full"},
        # a large single domain, eager launches
        {"name": "steps-512", "kind": "steps", "nx": 512, "ny": 512, "nz": 256, "grains": 16, "slots": 8, "steps": 10,
         "graph": False, "model": "full"},
        # a submitted job end to end: pinned field in, 10 steps, pinned field out
        {"name": "job-128", "kind": "job", "nx": 128, "ny": 128, "nz": 128, "grains": 32, "slots": 8, "steps": 10,
         "model": "full"},
        # batched bicrystals of the orientation study's sizes, replayed from a graph
        {"name": "batch-24", "kind": "batch", "instances": 24, "xy_max": 128, "z_max": 96, "steps": 20,
         "model": "full"},
        # observables of a headline-size state, sampled while a run advances
        {"name": "metrics-256", "kind": "metrics", "nx": 256, "ny": 256, "nz": 256, "grains": 64, "slots": 8},
        # surrogate: one optimiser step at the default batch
        {"name": "train-512", "kind": "train", "rows": 512},
        # surrogate: outputs of the whole candidate set
        {"name": "forward-65536", "kind": "forward", "rows": 65536},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi, most):
    """A box of sides lo..hi, odd ones among them, of at most `most` cells."""
    while True:
        d = [_log_int(rng, lo, hi) for _ in range(3)]
        if rng.random() < 0.4:
            d = [max(lo, v // 4 * 4) for v in d]
        if d[0] * d[1] * d[2] <= most:
            # grains of about 8^3 cells and more in the slab, as in the listed boxes
            grains = min(_log_int(rng, 1, 64), max(1, d[0] * d[1] * max(8, d[2] // 8) // 512))
            return {"nx": d[0], "ny": d[1], "nz": d[2], "grains": grains}


def draw(rng):
    kind = rng.choice(["dropin", "dropin", "steps", "steps", "steps", "job", "batch", "metrics", "train", "forward"])
    if kind == "dropin":
        return {"kind": kind, **_box(rng, 24, 256, 1 << 23),
                "dtype": rng.choice(["float32", "float64"]), "checked": rng.random() < 0.5,
                "model": rng.choice(list(MODELS))}
    if kind == "steps":
        return {"kind": kind, **_box(rng, 24, 400, 1 << 24),
                "slots": rng.choice([8, 16]), "steps": rng.choice([2, 4, 10]), "graph": rng.random() < 0.5,
                "model": rng.choice(list(MODELS))}
    if kind == "job":
        return {"kind": kind, **_box(rng, 24, 160, 1 << 21),
                "slots": rng.choice([8, 16]), "steps": rng.choice([4, 10]), "model": rng.choice(list(MODELS))}
    if kind == "batch":
        return {"kind": kind, "instances": _log_int(rng, 2, 32), "xy_max": rng.choice([32, 64, 96, 128]),
                "z_max": rng.choice([64, 96]), "steps": rng.choice([10, 20]), "model": rng.choice(list(MODELS))}
    if kind == "metrics":
        return {"kind": kind, **_box(rng, 24, 256, 1 << 24),
                "slots": rng.choice([8, 16])}
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 32, 2048)}
    return {"kind": kind, "rows": _log_int(rng, 64, 65536)}


# -- inputs -----------------------------------------------------------------------------------

class Model:
    """Physical parameters of the reference's 3D configuration and what follows from them."""

    def __init__(self):
        self.dx, self.dt, self.T_melt, self.Sf = 1.0e-4, 5.0e-5, 1687.0, 2.12e4
        self.delta_a, self.mu_a, self.p_round, self.ksi = 0.36, 0.6156, 0.05, 0.05
        self.delta = 6.0 * self.dx
        self.eps0, self.eps_gb = (math.sqrt(8.0 * self.delta * g / math.pi ** 2) for g in (0.44, 0.60))
        self.w0, self.w_gb = 4.0 * 0.44 / self.delta, 4.0 * 0.60 / self.delta
        self.m_sl = math.pi ** 2 / (8.0 * self.delta) * 5.0e-5
        self.m_gb = self.m_sl * 0.07
        self.a0, self.theta_c = math.radians(54.7), math.radians(10.0)
        self.g2_floor = (0.1 / self.dx) ** 2
        self.gradient = 1.0e2
        self.cooling_rate = self.gradient * 5.0e-2 * self.dt

    def scalars(self, cast):
        """The 13 floating-point arguments of the update kernel."""
        return tuple(cast(v) for v in (self.dx, self.dt, self.T_melt, self.Sf, self.eps0, self.w0, self.a0,
                                       self.delta_a, self.mu_a, self.p_round, self.g2_floor, self.ksi, self.theta_c))

    def matrices(self, N):
        """wij, aij, mij [N, N] float32: phase 0 is the liquid."""
        out = []
        for sl, gb in ((self.w0, self.w_gb), (self.eps0, self.eps_gb), (self.m_sl, self.m_gb)):
            a = np.full((N, N), gb, np.float32)
            a[0, :] = a[:, 0] = sl
            np.fill_diagonal(a, 0.0)
            out.append(a)
        return out


MODEL = Model()


def _quats(rng, shape):
    q = rng.standard_normal(tuple(shape) + (4,))
    return q / np.linalg.norm(q, axis=-1, keepdims=True)


def _normals(quats):
    """[n, 8, 3] float32: the {111} normals rotated by unit quaternions (x, y, z, w)."""
    x, y, z, w = np.moveaxis(np.asarray(quats, np.float64), -1, 0)
    R = np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
                  np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
                  np.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], -2)
    base = np.array([[1, 1, 1], [1, 1, -1], [1, -1, 1], [-1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1],
                     [-1, -1, -1]], np.float64) / math.sqrt(3.0)
    first = R[:, None] @ base[None, :4, :, None]
    u = first[..., 0].astype(np.float32)
    return np.concatenate([u, -u[:, ::-1]], 1)  # 4 antipodal pairs


def _voronoi(case, seed):
    """A Voronoi slab of grains under a tanh front near the top of the slab."""
    rng = np.random.default_rng(seed)
    nx, ny, nz, G = case["nx"], case["ny"], case["nz"], case["grains"]
    slab = max(8, nz // 8)
    seeds = torch.from_numpy(rng.uniform(0.0, 1.0, (G, 3)) * [nx, ny, slab]).to(DEVICE, torch.float32)
    at = [torch.arange(n, device=DEVICE, dtype=torch.float32) for n in (nx, ny, slab)]
    d = []
    for a, n in ((0, nx), (1, ny), (2, 0)):
        e = (at[a][None] - seeds[:, a:a + 1]).abs()
        d.append((torch.minimum(e, n - e) if n else e) ** 2)
    best = torch.full((nx, ny, slab), math.inf, device=DEVICE)
    owner = torch.zeros((nx, ny, slab), dtype=torch.int32, device=DEVICE)
    for g in range(G):
        r = d[0][g][:, None, None] + d[1][g][None, :, None] + d[2][g][None, None, :]
        owner[r < best] = g + 1
        best = torch.minimum(best, r)
    height = slab + rng.uniform(-1.0, 1.0)
    prof = 0.5 * (1.0 - np.tanh(2.2 / MODEL.delta * (np.arange(nz) - height) * MODEL.dx))
    prof = prof.astype(np.float32)
    quats = np.concatenate([[[0.0, 0.0, 0.0, 1.0]], _quats(rng, (G,))])
    T0z = MODEL.T_melt + MODEL.gradient * (np.arange(nz) - slab) * MODEL.dx
    T0z = T0z.astype(np.float32).astype(np.float64)
    return owner, prof, T0z, _normals(quats)


def _dense(owner, prof, N, dtype, pinned=False):
    """Dense phi [N, nx, ny, nz] of an owner map and a solid-fraction profile."""
    nx, ny, slab = owner.shape
    nz = len(prof)
    s = torch.from_numpy(prof).to(DEVICE)
    phi = torch.zeros((N, nx, ny, nz), dtype=torch.float32, device=DEVICE)
    phi[0] = (1.0 - s).clamp(0.0, 1.0)
    phi[:, :, :, :slab].scatter_(0, owner[None].long(), s[:slab].expand(1, nx, ny, slab))
    if nz > slab:
        top = owner[:, :, -1:].long().expand(nx, ny, nz - slab)
        phi[:, :, :, slab:].scatter_(0, top[None], s[slab:].expand(1, nx, ny, nz - slab))
    phi = phi.to(dtype)
    return phi.cpu().pin_memory() if pinned else phi


def _solver(case, seed):
    from mpf3d.solver import CompactSolver

    owner, prof, T0z, n111 = _voronoi(case, seed)
    aniso, torque = MODELS[case.get("model", "full")]
    more = {"slots": case["slots"], "anisotropy": bool(aniso), "torque": bool(torque), "device": DEVICE}
    return CompactSolver.from_owner(owner.cpu().numpy(), prof, T0z, n111, *MODEL.matrices(case["grains"] + 1), **more)


def _start(sim):
    """A start state that a run can be brought back to: both buffers hold it, so that no record is unwritten."""
    for t in sim.buf[1]:
        t.zero_()
    return [t.clone() for t in sim.buf[0]]


def _restore(sim, start):
    for dst, src in zip(sim.buf[0], start):
        dst.copy_(src)
    sim.cur = sim.step_count = 0
    sim.forget_history()


def _batch_inputs(case, seed):
    rng = np.random.default_rng(case["instances"])  # the boxes belong to the case, what fills them to the seed
    xy = [v for v in (32, 48, 64, 96, 128) if case["xy_max"] / 2 <= v <= case["xy_max"]]
    dims = [(int(rng.choice(xy)), int(rng.choice(xy)), int(rng.choice([64, case["z_max"]])))
            for _ in range(case["instances"])]
    dims[0] = (case["xy_max"], case["xy_max"], case["z_max"])
    n, rng = len(dims), np.random.default_rng(seed)
    return dims, _quats(rng, (n, 2)), rng.uniform(0.25, 3.0, n), rng.uniform(0.0, 1.0, n)


def _rows(case, seed):
    """Network inputs [rows, 14] (two orientations, undercooling, anisotropy strength, facet alignments) and targets."""
    rng = np.random.default_rng(seed)
    M = case["rows"]
    q = _quats(rng, (M, 2))
    q = np.where(q[..., 3:] < 0, -q, q)
    up = np.sort(np.abs(_normals(q.reshape(-1, 4))[:, :4, 2].astype(np.float64)), 1)[:, :1:-1].reshape(M, 4)
    X = np.concatenate([q.reshape(M, 8), rng.uniform(-1.0, 1.0, (M, 2)), 2.0 * up - 1.0], 1).astype(np.float32)
    Y = np.stack([np.tanh(X[:, 8] * X[:, 10] + 0.3 * X[:, 12]), 0.5 * X[:, 9] - X[:, 0] * X[:, 5]], 1)
    return X, ((Y - Y.mean(0)) / (Y.std(0) + 1e-6)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        dt = getattr(torch, case["dtype"])
        owner, prof, T0z, n111 = _voronoi(case, seed)
        N = case["grains"] + 1
        phi = _dense(owner, prof, N, dt)
        shape = tuple(phi.shape[1:])
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)
        return {"case": case, "phi": phi, "phi_new": torch.zeros_like(phi),
                "temp": torch.from_numpy(T0z).to(DEVICE, dt).expand(shape).contiguous(),
                "mf": torch.zeros((50,) + shape, dtype=torch.int32, device=DEVICE),
                "nf": torch.zeros(shape, dtype=torch.int32, device=DEVICE),
                "status": torch.zeros(2, dtype=torch.int32, device=DEVICE),
                "mats": [dev(a) for a in MODEL.matrices(N)] + [dev(n111)],
                "scalars": MODEL.scalars(np.float32 if dt == torch.float32 else np.float64),
                "rate": (np.float32 if dt == torch.float32 else np.float64)(MODEL.cooling_rate)}
    if kind == "steps":
        sim = _solver(case, seed)
        state = {"case": case, "sim": sim, "start": _start(sim),
                 "phi": torch.empty((sim.N, sim.nx, sim.ny, sim.nz), dtype=torch.float32, device=DEVICE)}
        if case["graph"]:
            sim.capture(case["steps"])
        return state
    if kind == "job":
        owner, prof, T0z, n111 = _voronoi(case, seed)
        phi = _dense(owner, prof, case["grains"] + 1, torch.float32, pinned=True)
        return {"case": case, "phi": phi, "out": torch.empty(phi.shape, pin_memory=True), "T0z": T0z, "n111": n111,
                "mats": MODEL.matrices(case["grains"] + 1)}
    if kind == "batch":
        from mpf3d.batched import BatchedBicrystals

        aniso, torque = MODELS[case["model"]]
        dims, q, under, da = _batch_inputs(case, seed)
        sim = BatchedBicrystals(dims, q, under, da, anisotropy=bool(aniso), torque=bool(torque), device=DEVICE)
        state = {"case": case, "sim": sim, "start": _start(sim),
                 "phi": [torch.empty((3,) + d, device=DEVICE) for d in sim.dims]}
        sim.capture(case["steps"])
        return state
    if kind == "metrics":
        sim = _solver(case, seed)
        sim.step(10)  # the initial profile's tails are clipped: a state of a running simulation
        return {"case": case, "sim": sim}
    from mpf3d.surrogate import Surrogate

    X, Y = _rows(case, seed)
    net = Surrogate(seed=seed % 1000, device=DEVICE)
    return {"case": case, "net": net, "x": net.prepare(X), "y": torch.from_numpy(Y).to(DEVICE)}


# -- passes -----------------------------------------------------------------------------------

def _run_dropin(s):
    from src import gpu_kernels_3d as K

    case = s["case"]
    N, nx, ny, nz = s["phi"].shape
    dims = (nx, ny, nz, N)
    K.kernel_update_temp_3d[UPDATE_LAUNCH](s["temp"], s["rate"], nx, ny, nz)
    if case["checked"]:
        K.kernel_update_nfmf_3d_checked[UPDATE_LAUNCH](s["phi"], s["mf"], s["nf"], s["status"], *dims)
    else:
        K.kernel_update_nfmf_3d[UPDATE_LAUNCH](s["phi"], s["mf"], s["nf"], *dims)
    args = (s["phi"], s["phi_new"], s["temp"], s["mf"], s["nf"], *s["mats"], *dims, *s["scalars"])
    if case["checked"] or case["model"] != "full":
        aniso, torque = MODELS[case["model"]]
        K.kernel_update_phasefield_active_3d_switchable[UPDATE_LAUNCH](*args, np.int32(aniso), np.int32(torque))
    else:
        K.kernel_update_phasefield_active_3d[UPDATE_LAUNCH](*args)
    return {"phi": s["phi_new"], "mf": s["mf"], "nf": s["nf"], "status": s["status"], "temp": s["temp"]}


def _run_job(s):
    from mpf3d.solver import CompactSolver

    case = s["case"]
    aniso, torque = MODELS[case["model"]]
    sim = CompactSolver(s["phi"], s["T0z"], s["n111"], *s["mats"], slots=case["slots"], anisotropy=bool(aniso),
                        torque=bool(torque), device=DEVICE)
    sim.step(case["steps"])
    return sim.to_dense(out=s["out"])


def _run_batch(s):
    from mpf3d import _lib

    sim = s["sim"]
    _restore(sim, s["start"])
    sim.step(s["case"]["steps"])
    head, idx, val = sim.buf[sim.cur]
    stream = torch.cuda.current_stream().cuda_stream or None
    for i, (out, d) in enumerate(zip(s["phi"], sim.dims)):
        _lib.check(_lib.lib().mpf3d_compact_to_dense_view(
            head.data_ptr(), idx.data_ptr(), val.data_ptr(), sim.slots, sim.total_cells, sim.inst_host[i].offset, 3,
            *d, out.data_ptr(), 0, stream), "compact_to_dense_view")
    return s["phi"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dropin":
        return _run_dropin(state)
    if kind == "steps":
        sim = state["sim"]
        _restore(sim, state["start"])
        sim.step(case["steps"], check=not case["graph"])
        return sim.to_dense(out=state["phi"], host=False)
    if kind == "job":
        return _run_job(state)
    if kind == "batch":
        return _run_batch(state)
    if kind == "metrics":
        m = state["sim"].metrics()
        return {"metrics": {**m, "grain_volumes": np.asarray(m["grain_volumes"])},
                "front": state["sim"].interface_positions()}
    net = state["net"]
    if kind == "train":
        loss = net.loss_and_grad(state["x"], state["y"])
        net.adam(lr=2e-3)
        return {"loss": loss, "gradients": net.g, "weights": net.w}
    return net.forward(state["x"])


# -- what a pass cannot do without -----------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("train", "forward"):
        params, rows = 16 * 256 + 2 * 256 * 256 + 2 * 256 + 770, case["rows"]
        if kind == "forward":
            return {"bytes": rows * (32 + 8) + 2 * params, "flops": 2 * rows * params}
        return {"bytes": rows * (32 + 8) + params * (4 * 4 + 3 * 4 + 2 * 2), "flops": 6 * rows * params}
    if kind == "batch":
        side = 0.75 * case["xy_max"]
        cells, N = case["instances"] * side * side * 0.5 * (64 + case["z_max"]), 3
    else:
        cells, N = case["nx"] * case["ny"] * case["nz"], case["grains"] + 1
    if kind == "dropin":
        size = 4 if case["dtype"] == "float32" else 8
        return {"bytes": cells * (2 * N * size + 2 * size + 8), "flops": cells * 100}
    if kind == "metrics":
        return {"bytes": cells * 4.5, "flops": cells * 10}
    if kind == "batch":
        # about half of the cells hold two phases and change at every step
        return {"bytes": cells * (10 * case["steps"] + 28 + 4 * N), "flops": cells * 500 * case["steps"]}
    dense = 4 * N * cells * (2 if kind == "job" else 1)
    # heads of the cells near the front and the records of the changing tenth, each step
    return {"bytes": dense + cells * (28 + 3 * case["steps"]), "flops": cells * 100 * case["steps"]}


# -- the same results in 64 bits --------------------------------------------------------------

def _shift(a, axis, by):
    """Neighbour values along a space axis (last three): x, y periodic, z clamped."""
    if axis < 2:
        return torch.roll(a, -by, a.dim() - 3 + axis)
    return torch.cat([a[..., 1:], a[..., -1:]], -1) if by > 0 else torch.cat([a[..., :1], a[..., :-1]], -1)


def _facet(g, u, floor):
    """Best {111} normal of gradients g [..., 3]: (|g|^2 >= floor, signed cosine, normal)."""
    q = (g * g).sum(-1)
    dot = (g[..., None, :] * u).sum(-1) / q.clamp_min(1e-300).sqrt()[..., None]
    best = dot.abs().argmax(-1, keepdim=True)
    cos = dot.gather(-1, best)[..., 0].clamp(-1.0, 1.0)
    n = u.expand(dot.shape + (3,)).gather(-2, best[..., None].expand(best.shape + (3,)))[..., 0, :]
    ok = q >= floor
    return ok, torch.where(ok, cos, 0.0), n, q


def _exact_chunk(phi, grad, cells, act, dT, wij, aij, mij, u, delta_a, aniso, torque):
    """New fractions of the given cells' active phases: (ids [A, C], values [A, C], valid [A, C])."""
    P, (N, nx, ny, nz) = MODEL, phi.shape
    flat = phi.view(N, -1)
    l, m, k = cells // (ny * nz), cells // nz % ny, cells % nz
    at = lambda a, b, c: (a * ny + b) * nz + c
    xp, xm, yp, ym = (l + 1) % nx, (l - 1) % nx, (m + 1) % ny, (m - 1) % ny
    zp, zm = (k + 1).clamp(max=nz - 1), (k - 1).clamp(min=0)
    nb = torch.stack([cells, at(xp, m, k), at(xm, m, k), at(l, yp, k), at(l, ym, k), at(l, m, zp), at(l, m, zm)])
    key = torch.where(act, torch.arange(N, 0, -1, device=phi.device)[:, None], 0)
    A = int(act.sum(0).max())
    key = key.topk(A, 0).values
    ids, ok = (N - key).clamp(max=N - 1), key > 0
    n = ok.sum(0)
    v = torch.where(ok[None], flat[ids[None], nb[:, None]], 0.0)  # [7, A, C]
    lap = (v[1:].sum(0) - 6.0 * v[0]) / P.dx ** 2
    L = flat[0][nb]
    liq, sol = ok & (ids == 0), ok & (ids > 0)
    w_sl = torch.full_like(dT, P.w0)
    if aniso:
        a_of = lambda c: P.mu_a * (1.0 + delta_a * ((c * c + P.p_round ** 2).sqrt() + math.tan(P.a0) *
                                                    ((1.0 - c * c).clamp_min(0.0) + P.p_round ** 2).sqrt()))
        g = grad[:, nb].permute(1, 2, 0)  # [7, C, 3]
        lap_sl, b = torch.zeros_like(lap), torch.ones_like(lap)
        for t in range(A):
            valid, c, un, q = _facet(g, u[ids[t]][None], P.g2_floor)
            a = a_of(c.abs())
            e2 = (P.eps0 * a) ** 2
            s = sum((e2[0] + e2[p]) * (L[p] - L[0]) for p in range(1, 7)) / (2.0 * P.dx * P.dx)
            if torque:
                ig = q.clamp_min(1e-300).rsqrt()
                coef = c / (c * c + P.p_round ** 2).sqrt() - math.tan(P.a0) * c / (
                    (1.0 - c * c).clamp_min(0.0) + P.p_round ** 2).sqrt()
                dc = un * ig[..., None] - ((g * un).sum(-1) * ig ** 3)[..., None] * g
                da = torch.where(valid[..., None], P.mu_a * delta_a * coef[..., None] * dc, 0.0)
                lq = lambda i, j, h: flat[0][at(i, j, h)]
                qq = 0.25 / P.dx ** 2
                dd = [(L[1 + 2 * x] - 2.0 * L[0] + L[2 + 2 * x]) / P.dx ** 2 for x in range(3)]
                xy = (lq(xp, yp, k) - lq(xp, ym, k) - lq(xm, yp, k) + lq(xm, ym, k)) * qq
                xz = (lq(xp, m, zp) - lq(xp, m, zm) - lq(xm, m, zp) + lq(xm, m, zm)) * qq
                yz = (lq(l, yp, zp) - lq(l, yp, zm) - lq(l, ym, zp) + lq(l, ym, zm)) * qq
                H = [[dd[0], xy, xz], [xy, dd[1], yz], [xz, yz, dd[2]]]
                E = 0.0
                for x in range(3):
                    q_x = 2.0 * sum(g[0][:, j] * H[x][j] for j in range(3))
                    a_x = P.mu_a * delta_a * coef[0] * sum(dc[0][:, j] * H[x][j] for j in range(3))
                    div = (da[1 + 2 * x][:, x] - da[2 + 2 * x][:, x]) * (0.5 / P.dx)
                    E = E + a_x * da[0][:, x] * q[0] + a[0] * div * q[0] + a[0] * da[0][:, x] * q_x
                s = s + torch.where(valid[0], P.eps0 ** 2 * E, 0.0)
            lap_sl[t] = s
            theta = torch.acos(c[0].abs())
            y = (0.5 * math.pi * theta / P.theta_c).clamp(1e-6, 0.5 * math.pi - 1e-6)
            tn = torch.tan(y)
            b[t] = torch.where(theta >= P.theta_c, 1.0, P.ksi + (1.0 - P.ksi) * tn * torch.tanh(1.0 / tn))
        top = torch.where(sol, v[0], -1.0)
        i_s = top.argmax(0)
        pick = lambda x: x.gather(0, i_s[None])[0]
        gs = torch.stack([pick(v[1 + 2 * x] - v[2 + 2 * x]) / (2.0 * P.dx) for x in range(3)], -1)
        _, c, _, _ = _facet(gs, u[pick(ids)], P.g2_floor)
        w_sl = torch.where(sol.any(0), P.w0 * a_of(c.abs()) ** 2, P.w0)
    else:
        lap_sl, b = P.eps0 ** 2 * torch.where(liq, lap, 0.0).sum(0).expand_as(lap), torch.ones_like(lap)
    W, G = torch.zeros_like(lap), torch.zeros_like(lap)
    for i in range(A):
        for j in range(A):
            w = torch.where(liq[j] & sol[i], w_sl, wij[ids[i], ids[j]])
            W[i] += w * v[0, j]
            G[i] += aij[ids[i], ids[j]] ** 2 * lap[j]
    new = v[0].clone()
    for i in range(A):
        d = torch.zeros_like(dT)
        for j in range(A):
            if i == j:
                continue
            sl, ls = sol[i] & liq[j], liq[i] & sol[j]
            T = torch.where(sl, 0.5 * lap_sl[i], torch.where(ls, -0.5 * lap_sl[j], 0.5 * (G[i] - G[j])))
            force = 8.0 / 3.1415926535 * (v[0, i] * v[0, j]).clamp_min(0.0).sqrt() * P.Sf * dT * (
                ls.double() - sl.double())
            mob = mij[ids[i], ids[j]] * torch.where(sl, b[i], torch.where(ls, b[j], 1.0))
            d = d - torch.where(ok[i] & ok[j], 2.0 * mob / n * (W[i] - W[j] + T - force), 0.0)
        new[i] = torch.where(ok[i], new[i] + P.dt * d, 0.0)
    new = new.clamp(0.0, 1.0)
    total = new.sum(0)
    new = torch.where(total > 1e-20, new / total.clamp_min(1e-300), torch.where(liq, 1.0, new))
    return ids, new, ok


def _exact_steps(phi, dT_of, steps, mats, u, delta_a, model):
    """`steps` steps of the phase-field model on dense float64 phi; dT_of(step) gives T - T_melt over z."""
    aniso, torque = MODELS[model]
    N, nx, ny, nz = phi.shape
    for step in range(1, steps + 1):
        act = phi > 0
        act = act | _shift(act, 0, 1) | _shift(act, 0, -1) | _shift(act, 1, 1) | _shift(act, 1, -1) | \
            _shift(act, 2, 1) | _shift(act, 2, -1)
        count = act.sum(0, dtype=torch.int32).view(-1)
        grad = torch.stack([(_shift(phi[0], x, 1) - _shift(phi[0], x, -1)).view(-1) for x in range(3)])
        grad /= 2.0 * MODEL.dx
        new = torch.where(act & (count.view(nx, ny, nz) == 1), 1.0, 0.0).to(torch.float64)
        busy, dT = torch.nonzero(count > 1)[:, 0], dT_of(step)
        for part in busy.split(1 << 19):
            ids, val, ok = _exact_chunk(phi, grad, part, act.view(N, -1)[:, part], dT[part % nz], *mats, u, delta_a,
                                        aniso, torque)
            at = (ids * (nx * ny * nz) + part)[ok]
            new.view(-1)[at] = val[ok]
        phi = new
    return phi


def _double(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE, torch.float64) for a in arrays]


def _exact_net(case, seed):
    """The surrogate's initial weights [(W, b)], its inputs and its targets."""
    rng = np.random.default_rng(seed % 1000)
    layers = []
    for K, N in ((16, 256), (256, 256), (256, 256), (256, 2)):
        bound = 1.0 / math.sqrt(10 if K == 16 else K)
        W = rng.uniform(-bound, bound, (N, K)).astype(np.float32)
        if K == 16:
            W[:, 14:] = 0.0
        layers.append((W, rng.uniform(-bound, bound, N).astype(np.float32)))
    X, Y = _rows(case, seed)
    x = torch.zeros((len(X), 16), device=DEVICE)
    x[:, :14] = torch.from_numpy(X).to(DEVICE)
    return [[torch.from_numpy(a).to(DEVICE) for a in p] for p in layers], x.bfloat16().double(), _double(Y)[0]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "forward"):
        layers, h, y = _exact_net(case, seed)
        params = [[W.bfloat16().double().requires_grad_(), b.double().requires_grad_()] for W, b in layers]
        for i, (W, b) in enumerate(params):
            h = h @ W.T + b
            h = torch.nn.functional.silu(h) if i < 3 else h
        if kind == "forward":
            return h.detach()
        loss = ((h - y) ** 2).sum() / len(y)
        loss.backward()
        g = torch.cat([p.grad.reshape(-1) for layer in params for p in layer])
        w = torch.cat([p.double().reshape(-1) for layer in layers for p in layer])
        return {"loss": loss.detach().reshape(1), "gradients": g, "weights": w - 2e-3 * g / (g.abs() + 1e-8)}
    if kind == "metrics":
        return None  # its state is ten steps from the inputs: the steps have cases of their own
    if kind == "batch":
        dims, q, under, da = _batch_inputs(case, seed)
        out = []
        for i, (nx, ny, nz) in enumerate(dims):
            z = np.float32(np.float32(2.2 / MODEL.delta) * MODEL.dx) * (np.arange(nz) - 16.0)
            prof = (0.5 * (1.0 - np.tanh(z))).astype(np.float32)
            owner = torch.full((nx, ny, 1), 2, dtype=torch.int32, device=DEVICE)
            owner[:nx // 2] = 1
            u = _double(_normals(np.concatenate([[[0.0, 0.0, 0.0, 1.0]], q[i]])))[0]
            dT = torch.full((nz,), -float(under[i]), dtype=torch.float64, device=DEVICE)
            out.append(_exact_steps(_dense(owner, prof, 3, torch.float64), lambda step: dT, case["steps"],
                                    _double(*MODEL.matrices(3)), u, float(da[i]), case["model"]))
        return out
    if case["nx"] * case["ny"] * case["nz"] * case.get("steps", 1) > 4e8:
        return None
    owner, prof, T0z, n111 = _voronoi(case, seed)
    T0z, u = _double(T0z, n111)
    N = case["grains"] + 1
    phi = _exact_steps(_dense(owner, prof, N, torch.float64), lambda step: T0z - MODEL.T_melt - step * MODEL.cooling_rate,
                       case.get("steps", 1), _double(*MODEL.matrices(N)), u, MODEL.delta_a, case["model"])
    if kind != "dropin":
        return phi.cpu() if kind == "job" else phi
    return {"phi": phi, "mf": None, "nf": None, "status": None,
            "temp": (T0z - MODEL.cooling_rate).expand(phi.shape[1:]).contiguous()}
