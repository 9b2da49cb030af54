"""Performance cases: the solver's work as its users call it, over the sizes it is used at.

Five kinds of call, all through the package's public classes:

* ``gn``      ``BatchSolver.gn_step``: the reference's undamped Gauss-Newton step;
* ``lm``      ``BatchSolver.reset`` + ``iterate(n)``: n Levenberg-Marquardt iterations from a
              resident state, on a non-default stream (where they replay as a CUDA graph);
* ``solve``   ``BatchSolver.solve`` + ``get_state``: a whole solve and its readback;
* ``dropin``  the reference binding's class ``CudaSolver``: state in, ``step(k)``, state out;
* ``train``   ``learned.Controller.grad`` + ``adam_step``: a training step of the damping network.

Every pass first loads the initial state (a tracker hands over a new guess each time), so a
pass always does the same work.  What comes back are the poses and the inverse depths: as the
FP64 state of an FP64 solver, and rounded to float32 from a mixed-precision one (whose step is
formed from FP32 Jacobians; ``CudaSolver`` reads back float32 too).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import __graft_entry__

__graft_entry__.load_package()
from spgo_gb300 import learned  # noqa: E402
from spgo_gb300 import solver as sv  # noqa: E402
from spgo_gb300.problem import Problem  # noqa: E402

DEV = "cuda"
_stream = None  # the one stream that every solver here is driven on
F64 = torch.float64
FX, CX, CY, W_IMG, H_IMG, BASE = 500.0, 320.0, 240.0, 640.0, 480.0, float(np.float32(0.12))
EPS = float(np.float32(1e-4))                       # the solver's parameters are float32
ALPHA_MIN, ALPHA_MAX = float(np.float32(1.0 / 30.0)), float(np.float32(5.0))
LOSSES = {  # name: (loss, scale, near_boost)
    "l2": ("l2", 3.0, False),
    "huber": ("huber", 2.0, False),
    "reference": ("cauchy", 3.0, True),             # the reference kernel's own weights
}


def _case(kind, scene="circle", problems=1, poses=(10, 10), landmarks=(500, 500), precision="mixed", loss="l2",
          iterations=1, window=0, outliers=0.0):
    return {"kind": kind, "scene": scene, "problems": problems, "poses_min": poses[0], "poses_max": poses[1],
            "landmarks_min": landmarks[0], "landmarks_max": landmarks[1], "precision": precision, "loss": loss,
            "iterations": iterations, "window": window, "outliers": outliers}


def listed():
    cases = {
        # one small window (config 0's size), one Gauss-Newton step: the smallest call, all latency
        "window_gn": _case("gn", scene="corridor", loss="reference"),
        # the drop-in class: state written pose by pose, four steps, state read back
        "dropin_steps": _case("dropin", scene="corridor", loss="reference", iterations=4),
        # one sliding window of a running tracker, two damped iterations
        "window_lm": _case("lm", poses=(20, 20), landmarks=(1600, 1600), iterations=2),
        # config 0: a plain FP64 solve of one window to convergence, readback included
        "window_fp64_solve": _case("solve", precision="fp64", iterations=10),
        # the divergence study: 100 trials of the reference's window size stepped together
        "trials100_gn": _case("gn", problems=100, landmarks=(960, 960), loss="reference"),
        # the benchmark batch: 256 uneven windows, two damped iterations
        "windows256_lm": _case("lm", problems=256, poses=(8, 32), landmarks=(200, 3000), iterations=2),
        # the same batch on the plain FP64 path
        "windows256_fp64": _case("lm", problems=256, poses=(8, 32), landmarks=(200, 3000), precision="fp64"),
        # a whole mixed-precision solve of a batch under a Huber loss (20 iterations), readback included
        "windows64_solve": _case("solve", scene="corridor", problems=64, poses=(8, 32), landmarks=(400, 3000),
                                 loss="huber", iterations=20),
        # one large problem (config 1), both precisions: the factorisation over many blocks
        "corridor100_lm": _case("lm", scene="corridor", poses=(100, 100), landmarks=(20000, 20000), iterations=2),
        "corridor100_fp64": _case("lm", scene="corridor", poses=(100, 100), landmarks=(20000, 20000),
                                  precision="fp64"),
        # the largest: config 2, a covisibility window, outliers under a Huber loss
        "corridor500_lm": _case("lm", scene="corridor", poses=(500, 500), landmarks=(200000, 200000), loss="huber",
                                window=20, outliers=0.05),
        # one training step of the damping network at its default batch
        "train_step": {"kind": "train", "samples": 512},
    }
    return [dict(c, name=n) for n, c in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.08:
        return {"kind": "train", "samples": _log_int(rng, 64, 4096)}
    if pick < 0.28:  # one large problem
        poses = _log_int(rng, 60, 400)
        fp64 = poses <= 150 and rng.random() < 0.3
        return _case("lm", scene="corridor", poses=(poses, poses), landmarks=(poses * rng.randint(100, 400),) * 2,
                     precision="fp64" if fp64 else "mixed", loss=rng.choice(["l2", "huber"]),
                     iterations=1 if fp64 or poses > 200 else rng.randint(1, 2), window=rng.choice([0, 20]),
                     outliers=0.05 if rng.random() < 0.5 else 0.0)
    if pick < 0.36:
        poses = rng.randint(6, 16)
        return _case("dropin", scene="corridor", poses=(poses, poses), landmarks=(poses * rng.randint(30, 96),) * 2, loss="reference",
                     iterations=rng.randint(1, 6))
    # batches of windows, no larger than the benchmark's
    lo = rng.randint(6, 24)
    hi = lo + rng.randint(0, 12)
    lm_lo = rng.randint(25, 60) * hi
    lm_hi = lm_lo + rng.randint(0, 1500)
    problems = _log_int(rng, 1, max(1, min(256, 400000 // lm_hi)))
    kind = rng.choice(["gn", "lm", "lm", "lm", "solve"])
    if kind == "gn":
        return _case("gn", scene="corridor", problems=problems, poses=(lo, hi), landmarks=(lm_lo, lm_hi), loss="reference",
                     iterations=1, precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "lm":
        fp64 = rng.random() < 0.25
        return _case("lm", scene=rng.choice(["circle", "corridor"]), problems=problems, poses=(lo, hi),
                     landmarks=(lm_lo, lm_hi), precision="fp64" if fp64 else "mixed", loss=rng.choice(["l2", "huber"]),
                     iterations=1 if fp64 else rng.randint(1, 2))
    return _case("solve", scene="corridor", problems=min(problems, 48), poses=(lo, hi), landmarks=(lm_lo, lm_hi),
                 loss="huber", iterations=20)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _sizes(case):
    """(poses, landmarks) of every problem of a case, the same for every seed."""
    n = case["problems"]
    r = np.random.default_rng([n, case["poses_max"], case["landmarks_max"]])
    return list(zip(r.integers(case["poses_min"], case["poses_max"] + 1, n).tolist(),
                    r.integers(case["landmarks_min"], case["landmarks_max"] + 1, n).tolist()))


def _look(c, target):
    z = target - c
    z = z / z.norm(dim=-1, keepdim=True)
    x = torch.linalg.cross(torch.tensor([0.0, 1.0, 0.0], dtype=F64).expand_as(z), z)
    x = x / x.norm(dim=-1, keepdim=True)
    T = torch.eye(4, dtype=F64).repeat(len(c), 1, 1)
    T[:, :3, :3] = torch.stack([x, torch.linalg.cross(z, x), z], -1)
    T[:, :3, 3] = c
    return T


def _inv(T):
    out = torch.zeros_like(T)
    Rt = T[..., :3, :3].transpose(-1, -2)
    out[..., :3, :3] = Rt
    out[..., :3, 3] = -(Rt @ T[..., :3, 3:])[..., 0]
    out[..., 3, 3] = 1.0
    return out


def _skew(v):
    z = torch.zeros_like(v[..., 0])
    return torch.stack([z, -v[..., 2], v[..., 1], v[..., 2], z, -v[..., 0], -v[..., 1], v[..., 0], z],
                       -1).reshape(v.shape + (3,))


def _exp(xi):
    """SE(3) exponential of [n, 6] twists (rotation first)."""
    w, rho = xi[:, :3], xi[:, 3:]
    t2 = (w * w).sum(-1).clamp_min(1e-300)
    t = t2.sqrt()
    small = t < 1e-3
    ts = torch.where(small, torch.ones_like(t), t)
    a = torch.where(small, 1 - t2 / 6 + t2 * t2 / 120, torch.sin(ts) / ts)[:, None, None]
    b = torch.where(small, 0.5 - t2 / 24 + t2 * t2 / 720, (1 - torch.cos(ts)) / (ts * ts))[:, None, None]
    c = torch.where(small, 1 / 6 - t2 / 120 + t2 * t2 / 5040, (ts - torch.sin(ts)) / ts ** 3)[:, None, None]
    S = _skew(w)
    S2 = S @ S
    eye = torch.eye(3, dtype=xi.dtype, device=xi.device)
    T = torch.zeros(len(xi), 4, 4, dtype=xi.dtype, device=xi.device)
    T[:, :3, :3] = eye + a * S + b * S2
    T[:, :3, 3] = ((eye + b * S + c * S2) @ rho[:, :, None])[..., 0]
    T[:, 3, 3] = 1.0
    return T


def _scene(case, seed, N, L):
    """One synthetic stereo window: cameras on a circle facing its centre, or a sinusoidal
    path looking sideways; 1 px noise, perturbed poses and inverse depths."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    uni = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=F64)       # noqa: E731
    nrm = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=F64)      # noqa: E731
    F = N + 1
    k = torch.arange(F, dtype=F64)
    circle = case["scene"] == "circle"
    if circle:
        th = 2 * math.pi * k / F
        c = torch.stack([5 * torch.sin(th), 0 * k, -5 * torch.cos(th)], -1)
        W = _look(c, torch.zeros(3, dtype=F64))
        M = 2 * L + 64
        pts = uni(M, 3) * 10 - 5
        cand = torch.arange(F, device=DEV).expand(M, F)
    else:
        x = 0.3 * k
        c = torch.stack([x, 0 * k, 0.5 * torch.sin(2 * math.pi * x / 15)], -1)
        yaw = 0.15 * torch.cos(2 * math.pi * x / 15)
        W = _look(c, c + torch.stack([torch.sin(yaw), 0 * yaw, torch.cos(yaw)], -1))
        M = 2 * L + 64 if N < 60 else L + L // 4 + 64
        margin = 4.0 if N >= 60 else 1.5
        pts = uni(M, 3) * torch.tensor([0.3 * N + 2 * margin, 4.0, 4.5], device=DEV, dtype=F64) \
            + torch.tensor([-margin, -2.0, 3.5], device=DEV, dtype=F64)
        near = (pts[:, 0] / 0.3).round().long().clamp(0, F - 1)
        cand = near[:, None] + torch.arange(-27, 28, device=DEV)
    ok = (cand >= 0) & (cand < F)
    fr = cand.clamp(0, F - 1)
    W = (_inv(W[:1]) @ W).to(DEV)      # frame 0 is the world frame
    pts = ((pts - c[0].to(DEV)) @ _look(c[:1], (torch.zeros(1, 3, dtype=F64) if circle else
           c[:1] + torch.stack([torch.sin(yaw), 0 * yaw, torch.cos(yaw)], -1)[:1]))[0, :3, :3].to(DEV))
    R, t = W[:, :3, :3], W[:, :3, 3]
    pl = torch.einsum("mcji,mcj->mci", R[fr], pts[:, None] - t[fr])
    z = pl[..., 2]
    zs = torch.where(z.abs() > 1e-9, z, torch.full_like(z, 1e-9))
    ul, v, ur = FX * pl[..., 0] / zs + CX, FX * pl[..., 1] / zs + CY, FX * (pl[..., 0] - BASE) / zs + CX
    vis = ok & (z >= 0.5) & (z <= 30) & (v >= 0) & (v < H_IMG)
    vis &= (ul >= 0) & (ul < W_IMG) & (ur >= 0) & (ur < W_IMG)
    keep = (vis.sum(1) >= 2).nonzero()[:L, 0]
    if len(keep) < L:
        raise ValueError("too few visible landmarks")
    vis, fr, pts, z = vis[keep], fr[keep], pts[keep], z[keep]
    uv = torch.stack([ul, v, ur, v], -1)[keep]
    pickd = (uni(L) * vis.sum(1)).long()
    slot = (vis & (vis.cumsum(1) - 1 == pickd[:, None])).long().argmax(1)
    host = fr.gather(1, slot[:, None])[:, 0]
    alpha = 1.0 / z.gather(1, slot[:, None])[:, 0]
    if case["window"]:
        vis &= (fr - host[:, None]).abs() <= case["window"] // 2
    lm, col = vis.nonzero(as_tuple=True)                   # landmark-major, frames ascending
    frame = fr[lm, col]
    obs = uv[lm, col] + nrm(len(lm), 4)
    at_host = frame == host[lm]
    if case["outliers"]:
        bad = (~at_host & (uni(len(lm)) < case["outliers"])).nonzero()[:, 0]
        obs[bad] = uni(len(bad), 4) * torch.tensor([W_IMG, H_IMG, W_IMG, H_IMG], device=DEV, dtype=F64)
    obs = obs.float().double()                             # pixels come as float32 values
    ax = nrm(F, 3)
    d = torch.cat([0.01 * ax / ax.norm(dim=1, keepdim=True), 0.02 * nrm(F, 3)], 1)   # a tracker's guess
    d[0] = 0
    Wi = W @ _exp(d)
    inc = _inv(Wi[1:]) @ Wi[:-1]
    alpha0 = (alpha * (1 + 0.05 * nrm(L))).clamp(ALPHA_MIN, ALPHA_MAX)
    ptr = torch.zeros(L + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = vis.sum(1).cumsum(0)
    T_rl = np.eye(4)
    T_rl[0, 3] = BASE
    n = lambda x: x.cpu().numpy()                          # noqa: E731
    return Problem(n_poses=N, intrinsics=np.array([FX, FX, CX, CY] * 2), T_rl=T_rl, host=n(host.int()),
                   anchor_uv=n(obs[at_host][:, :2]).copy(), obs_ptr=n(ptr), obs_frame=n(frame.int()), obs_uv=n(obs),
                   poses=n(inc), alpha=n(alpha0))


def _problems(case, seed):
    return [_scene(case, 1000 * int(seed) + i, N, L) for i, (N, L) in enumerate(_sizes(case))]


def _training(case, seed):
    """Standardised-feature traces and an optimiser state some way into a training run."""
    r = np.random.default_rng([int(seed), 29])
    n = case["samples"]
    X = r.normal(size=(n, 16)).astype(np.float32)
    T = np.stack([r.choice([-6.0, -4.0, -3.0, -2.0, -1.0, 0.0, 1.0, 2.0, 3.0], n), r.integers(0, 2, n)],
                 1).astype(np.float32)
    theta = learned.init_params(int(seed) % 1000)
    m = (0.01 * r.normal(size=theta.size)).astype(np.float32)
    v = (1e-3 * (0.5 + r.random(theta.size))).astype(np.float32)
    return X, T, theta, m, v


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "train":
        X, T, theta, m, v = _training(case, seed)
        ctl = learned.Controller(theta, device=DEV)
        ctl.m.copy_(torch.from_numpy(m))
        ctl.v.copy_(torch.from_numpy(v))
        ctl.step = 100
        return {"case": case, "ctl": ctl, "X": X, "T": T}
    probs = _problems(case, seed)
    loss, scale, near = LOSSES[case["loss"]]
    if case["kind"] == "dropin":
        return _prepare_dropin(case, probs[0])
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    stream = _stream
    with torch.cuda.stream(stream):
        bs = sv.BatchSolver(probs, precision=case["precision"], device=DEV, stream=stream)
        bs.set_params(loss=loss, loss_scale=scale, near_boost=near, max_iters=case["iterations"],
                      tol=_tol(case))
        start = (bs.poses.clone(), bs.alpha.clone())
    return {"case": case, "bs": bs, "start": start, "stream": stream}


def _tol(case):
    """Stopping threshold: the library's own for FP64; a mixed solve runs out its budget of
    iterations (where it stops by the threshold depends on the last bits of the cost)."""
    return 1e-6 if case["precision"] == "fp64" else 1e-12


def _prepare_dropin(case, p):
    N, L = p.n_poses, p.n_landmarks
    M = -(-L // N)
    cs = sv.CudaSolver(N, M, device=DEV)
    cs.loadCalibration(p.intrinsics.reshape(4, 2), p.T_rl)
    lm = np.repeat(np.arange(L), np.diff(p.obs_ptr))
    left = np.ones((p.n_obs, 3), np.float32)
    right = left.copy()
    left[:, :2], right[:, :2] = p.obs_uv[:, :2], p.obs_uv[:, 2:]
    for o in range(p.n_obs):
        cs.writeObservations(p.host[lm[o]], p.obs_frame[o], lm[o], left[o], right[o])
    cs.setStepSize(0.5)
    alpha = np.ones(N * M, np.float32)
    alpha[:L] = p.alpha
    return {"case": case, "cs": cs, "poses": p.poses.astype(np.float32), "alpha": alpha}


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        ctl = state["ctl"]
        loss, grad = ctl.grad(state["X"], state["T"])
        ctl.adam_step(grad, 1e-3)
        return {"grad": grad, "theta": ctl.theta.clone()}
    if case["kind"] == "dropin":
        cs = state["cs"]
        for k, T in enumerate(state["poses"]):
            cs.writeIncrementalPose(k, T)
        cs.loadInverseDepths(state["alpha"])
        cs.step(case["iterations"])
        return {"poses": np.stack([cs.getIncrementalPose(k) for k in range(len(state["poses"]))]),
                "alpha": cs.getInverseDepths()}
    bs = state["bs"]
    with torch.cuda.stream(state["stream"]):
        bs.poses.copy_(state["start"][0])
        bs.alpha.copy_(state["start"][1])
        if case["kind"] == "solve":
            costs = np.array([s["cost"] for s in bs.solve()])
            poses, alpha = bs.get_state()
            out = {"poses": np.concatenate(poses)[:, :3].reshape(-1), "alpha": np.concatenate(alpha), "cost": costs}
            return out if case["precision"] == "fp64" else {k: v.astype(np.float32) for k, v in out.items()}
        if case["kind"] == "gn":
            bs.gn_step(case["iterations"], 1.0)
        else:
            bs.reset()
            bs.iterate(case["iterations"])
        if case["precision"] == "fp64":
            return {"poses": bs.poses, "alpha": bs.alpha}
        return {"poses": bs.poses.float(), "alpha": bs.alpha.float()}


def work(case):
    """Bytes and flops one pass cannot do without: per evaluation of the cost every
    observation (pixels, frame, landmark) and the state once; per linearisation its
    Jacobian products, the landmarks' elimination and the reduced system's factor."""
    if case["kind"] == "train":
        n, params = case["samples"], 5378
        return {"bytes": 4 * (n * 18 + 8 * params), "flops": 6.0 * n * params}
    N = (case["poses_min"] + case["poses_max"]) / 2
    L = (case["landmarks_min"] + case["landmarks_max"]) / 2
    span = N if case["scene"] == "circle" else min(N, case["window"] or 22)   # poses a landmark's window covers
    seen = (0.44 if case["scene"] == "circle" else 0.75 if case["window"] else 0.9) * (span + 1)
    B, it = case["problems"], case["iterations"]
    if case["kind"] == "solve" and case["precision"] == "fp64":
        it = 6                                                                # about what it converges in
    sweeps = it if case["kind"] in ("gn", "dropin") else it + 1
    per = 25.0 * seen * L + 40.0 * L + 200.0 * N                              # bytes
    flops = 400.0 * seen * L + (6 * span) ** 2 * L + (6 * N) * (6 * min(N, span)) ** 2 / 3
    return {"bytes": B * (sweeps * per + 16.0 * L + 200.0 * N), "flops": B * it * flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------

class _Exact:
    """One problem's FP64 state, cost, linearisation and damped step in plain torch."""

    def __init__(self, p, loss):
        d = lambda x, t=F64: torch.as_tensor(np.ascontiguousarray(x), device=DEV).to(t)  # noqa: E731
        self.N, self.L = p.n_poses, p.n_landmarks
        self.kind, self.scale, self.near = LOSSES[loss]
        self.host = d(p.host, torch.int64)
        self.lm = torch.repeat_interleave(torch.arange(self.L, device=DEV), d(np.diff(p.obs_ptr), torch.int64))
        self.n, self.uv = d(p.obs_frame, torch.int64), d(p.obs_uv)
        self.a = self.host[self.lm]
        pa = d(p.anchor_uv)
        self.ray = torch.stack([(pa[:, 0] - CX) / FX, (pa[:, 1] - CY) / FX, torch.ones_like(pa[:, 0])], -1)
        self.beta = torch.where((self.n - self.a).abs() < 2, 16.0, 1.0).to(F64) if self.near else 1.0
        self.poses, self.alpha = d(p.poses), d(p.alpha)
        order = torch.argsort(self.host, stable=True).cpu()
        self.groups = order.split(4096)
        self.rows = self._rows()

    def _rows(self):
        rows = []
        slot = torch.empty(self.L, dtype=torch.int64, device=DEV)
        for q in self.groups:
            q = q.to(DEV)
            mark = torch.zeros(self.L, dtype=torch.bool, device=DEV)
            mark[q] = True
            slot[q] = torch.arange(len(q), device=DEV)
            o = mark[self.lm].nonzero()[:, 0]
            lo = int(min(self.n[o].min(), self.host[q].min()))
            hi = int(max(self.n[o].max(), self.host[q].max()))
            rows.append((q, o, slot[self.lm[o]].clone(), lo, hi))
        return rows

    def chain(self, poses):
        G = [np.eye(4)]
        for T in poses.cpu().numpy():
            G.append(G[-1] @ np.linalg.inv(T))
        return torch.as_tensor(np.stack(G), device=DEV)

    def camera(self, poses, alpha):
        G = self.chain(poses)
        R, c = G[:, :3, :3], G[:, :3, 3]
        dX = torch.einsum("lij,lj->li", R[self.host], self.ray)       # world ray of each landmark
        X = c[self.host] + dX / alpha[:, None]
        res, pts, s = [], [], []
        t = torch.einsum("oji,oj->oi", R[self.n], X[self.lm] - c[self.n])
        for cam in (0, 1):
            q = t - torch.tensor([BASE * cam, 0, 0], device=DEV, dtype=F64)
            pr = FX * q[:, :2] / q[:, 2:] + torch.tensor([CX, CY], device=DEV, dtype=F64)
            res.append(self.uv[:, 2 * cam:2 * cam + 2] - pr)
            pts.append(q)
            s.append((res[-1] ** 2).sum(-1))
        return R, c, X, dX, res, pts, s

    def weights(self, s):
        if self.kind == "l2":
            return torch.ones_like(s) * self.beta, s * self.beta
        if self.kind == "cauchy":
            c2 = self.scale ** 2
            return self.beta / (1 + s / c2), self.beta * c2 * torch.log1p(s / c2)
        rs = s.sqrt()
        inl = rs <= self.scale
        return torch.where(inl, 1.0, self.scale / rs.clamp_min(1e-300)), \
            torch.where(inl, s, 2 * self.scale * rs - self.scale ** 2)

    def cost(self, poses, alpha):
        return 0.5 * sum(float(self.weights(s)[1].sum()) for s in self.camera(poses, alpha)[-1])

    def linearise(self):
        R, c, X, dX, res, pts, s = self.camera(self.poses, self.alpha)
        N, L = self.N, self.L
        C = torch.zeros(L, dtype=F64, device=DEV)
        ga = torch.zeros_like(C)
        lo, hi = torch.minimum(self.a, self.n), torch.maximum(self.a, self.n)
        sg = torch.where(self.n > self.a, 1.0, -1.0).to(F64) * (self.n != self.a)
        pair = torch.zeros(N + 1, N + 1, 42, dtype=F64, device=DEV).reshape(-1, 42)
        qj = torch.zeros(len(self.lm), 6, dtype=F64, device=DEV)
        gw = -dX / self.alpha[:, None] ** 2                            # dX / d alpha
        for cam in (0, 1):
            w2 = self.weights(s[cam])[0]
            x, y, z = pts[cam].unbind(-1)
            zero = torch.zeros_like(z)
            for row, jp in enumerate((torch.stack([FX / z, zero, -FX * x / z ** 2], -1),
                                      torch.stack([zero, FX / z, -FX * y / z ** 2], -1))):
                k = torch.einsum("oij,oj->oi", R[self.n], jp)          # d pixel / d world point
                r = res[cam][:, row]
                j = (k * gw[self.lm]).sum(-1)
                C.index_add_(0, self.lm, w2 * j * j)
                ga.index_add_(0, self.lm, w2 * j * r)
                q = torch.cat([k, torch.linalg.cross(X[self.lm], k)], -1)
                v = torch.cat([(w2[:, None, None] * q[:, :, None] * q[:, None, :]).reshape(-1, 36) * (sg * sg)[:, None],
                               (w2 * r * sg)[:, None] * q], -1)
                pair.index_add_(0, lo * (N + 1) + hi, v)
                qj += (w2 * j * sg)[:, None] * q
        # pose i's Jacobian row: q^T M_i over the observations whose range [lo, hi) holds i
        M = torch.zeros(N, 6, 6, dtype=F64, device=DEV)
        M[:, :3, :3] = _skew(c[:N]) @ R[:N]
        M[:, :3, 3:] = R[:N]
        M[:, 3:, :3] = R[:N]
        F = pair.reshape(N + 1, N + 1, 42).cumsum(0).flip(1).cumsum(1).flip(1)   # sums over lo <= i, hi >= j
        i, j = torch.triu_indices(N, N, device=DEV)
        blk = M[i].transpose(1, 2) @ F[i, j + 1, :36].reshape(-1, 6, 6) @ M[j]
        A = torch.zeros(N, N, 6, 6, dtype=F64, device=DEV)
        A[j, i] = blk.transpose(1, 2)
        A[i, j] = blk
        k = torch.arange(N, device=DEV)
        g = (M.transpose(1, 2) @ F[k, k + 1, 36:, None])[..., 0].reshape(-1)
        self.A, self.g, self.C, self.ga, self.M, self.qj = A.permute(0, 2, 1, 3).reshape(6 * N, 6 * N), g, C, ga, M, qj
        return self

    def columns(self):
        """The pose / inverse-depth block B, as (landmarks, first row, [rows, landmarks])."""
        for q, o, slot, lo, hi in self.rows:
            w = hi - lo + 1
            U = torch.zeros(len(q) * w, 6, dtype=F64, device=DEV)
            U.index_add_(0, slot * w + self.n[o] - lo, self.qj[o])
            U = U.reshape(len(q), w, 6)
            f = torch.arange(lo, hi, device=DEV)
            after = (U.sum(1, keepdim=True) - U.cumsum(1))[:, :-1]      # targets beyond pose i
            before = U.cumsum(1)[:, :-1]                                # targets up to pose i
            fwd = (f[None] >= self.host[q][:, None])[..., None]
            hostslot = (self.host[q] - lo)
            own = torch.zeros_like(U)
            own[torch.arange(len(q), device=DEV), hostslot] = 1
            b = torch.where(fwd, after, before)
            yield q, 6 * lo, torch.einsum("lfa,fab->fbl", b, self.M[lo:hi]).reshape(6 * (hi - lo), len(q))

    def step(self, lam):
        D = self.C * (1 + lam) + EPS
        dA = self.A.diagonal()
        S = self.A + torch.diag(lam * dA)
        gS = self.g.clone()
        for q, r, Bq in self.columns():
            s = slice(r, r + Bq.shape[0])
            S[s, s] -= (Bq / D[q]) @ Bq.T
            gS[s] -= Bq @ (self.ga[q] / D[q])
        Lc, info = torch.linalg.cholesky_ex(S)
        if int(info):
            return None
        d = torch.cholesky_solve(gS[:, None], Lc)[:, 0]
        da = torch.empty_like(self.C)
        for q, r, Bq in self.columns():
            da[q] = (self.ga[q] - Bq.T @ d[r:r + Bq.shape[0]]) / D[q]
        pred = 0.5 * float(d @ (self.g + lam * dA * d) + da @ (self.ga + (D - self.C) * da))
        return d, da, pred

    def moved(self, d, da, size):
        return self.poses @ _exp(size * d.reshape(-1, 6)), (self.alpha + da).clamp(ALPHA_MIN, ALPHA_MAX)

    def gauss_newton(self, n, size):
        for _ in range(n):
            d, da, _pred = self.linearise().step(0.0)
            self.poses, self.alpha = self.moved(d, da, size)

    def levenberg(self, n, tol):
        lam, nu = 1e-4, 2.0
        self.F = self.cost(self.poses, self.alpha)
        self.linearise()
        for _ in range(n):
            st = self.step(lam)
            rho = -1.0
            if st is not None:
                new = self.moved(st[0], st[1], 1.0)
                Fn = self.cost(*new)
                rho = (self.F - Fn) / st[2] if st[2] > 0 and math.isfinite(Fn) else -1.0
            if rho > 0:
                rel, self.F = (self.F - Fn) / self.F, Fn
                self.poses, self.alpha = new
                lam, nu = lam * max(1 / 3, 1 - (2 * rho - 1) ** 3), 2.0
                if rel < tol:
                    return
                self.linearise()
            else:
                lam, nu = lam * nu, nu * 2


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "solve" and case["precision"] != "fp64":
        return None          # at the noise floor a mixed solve rejects other steps than a 64-bit one
    poses, alpha, cost = [], [], []
    for p in _problems(case, seed):
        if case["kind"] == "dropin":   # the class takes its state as float32
            p.poses, p.alpha = p.poses.astype(np.float32), p.alpha.astype(np.float32)
        e = _Exact(p, case["loss"])
        if case["kind"] in ("gn", "dropin"):
            e.gauss_newton(case["iterations"], 0.5 if case["kind"] == "dropin" else 1.0)
        else:
            e.levenberg(case["iterations"], _tol(case))
            cost.append(e.F)
        poses.append(e.poses)
        alpha.append(e.alpha)
    if case["kind"] == "dropin":
        N = len(poses[0])
        rest = torch.ones(N * (-(-len(alpha[0]) // N)) - len(alpha[0]), dtype=F64, device=DEV)
        return {"poses": poses[0], "alpha": torch.cat([alpha[0], rest])}
    out = {"poses": torch.cat(poses)[:, :3].reshape(-1), "alpha": torch.cat(alpha)}
    if case["kind"] == "solve":
        out["cost"] = np.array(cost)
    return out


def _exact_train(case, seed):
    X, T, theta, m, v = (torch.from_numpy(x).to(F64) for x in _training(case, seed))
    theta.requires_grad_(True)
    parts, o = [], 0
    for shape in ((64, 16), (64,), (64, 64), (64,), (2, 64), (2,)):
        n = math.prod(shape)
        parts.append(theta[o:o + n].reshape(shape))
        o += n
    h = torch.nn.functional.gelu(X @ parts[0].T + parts[1])
    h = torch.nn.functional.gelu(h @ parts[2].T + parts[3])
    y = h @ parts[4].T + parts[5]
    loss = ((y[:, 0] - T[:, 0]) ** 2).mean() \
        + torch.nn.functional.binary_cross_entropy_with_logits(y[:, 1], T[:, 1])
    g, = torch.autograd.grad(loss, theta)
    m, v, t = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g, 101
    new = theta.detach() - 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return {"grad": g, "theta": new}
