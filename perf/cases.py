"""Workloads for timing the library through its public entry points.

Every case is work that a program using the library has it do, over the
sizes of the library's own configurations and benchmark:

  * the step on a state that the host keeps (one call per step);
  * the step loop on a state that the device keeps (one call per write
    interval: the plain steps, the write step and its energy row, then the
    state back on the host), in the three arithmetic modes;
  * the force pass on the caller's own device buffers;
  * the batched solver on a sweep of collisions, exact and double-float;
  * the surrogate network: prediction, gradients, training.

Clusters come from the library's seeded builder, pulled together by 1% so
that about one pair in twenty neighbours is in contact, as in the middle of
a collision.  ``exact`` restates the step and the network in plain torch, in
64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spacelab_gb300 import _lib, batch, configs
from spacelab_gb300.ball_group import BallGroup, GpuStep
from spacelab_gb300.surrogate import Mlp

SQUEEZE = 0.99  # positions of a built cluster are scaled by this: contacts of up to 1% of a diameter
NET = {"n_in": 8, "n_out": 4, "hidden": 256, "layers": 4}


def listed() -> list[dict]:
    return [
        # a host program that owns the arrays of a small aggregate and steps it call by call
        {"name": "host_step_exact_n96", "kind": "host_step", "mode": "exact", "n": 96, "shape": "cluster"},
        # the same program on the aggregate collision of the benchmark: one call per step
        {"name": "host_step_exact_n5000", "kind": "host_step", "mode": "exact", "n": 5000, "shape": "collision"},
        # the 1000-sphere dust cluster, one write interval of 100 steps
        {"name": "loop_exact_n1000", "kind": "loop", "mode": "exact", "n": 1000, "shape": "cluster", "skip": 100},
        # the polydisperse cluster in FP64, a short write interval: the largest system of the configurations
        {"name": "loop_exact_n20000", "kind": "loop", "mode": "exact", "n": 20000, "shape": "polydisperse",
         "skip": 20},
        # the same cluster in the two mixed forms
        {"name": "loop_mixed_n20000", "kind": "loop", "mode": "mixed", "n": 20000, "shape": "polydisperse",
         "skip": 20},
        # one collision of the sweep run alone, of an odd size, in the double-float form
        {"name": "loop_mixed_df_n1733", "kind": "loop", "mode": "mixed_df", "n": 1733, "shape": "collision",
         "skip": 100},
        # the force pass of a host application on its own device buffers
        {"name": "static_n201", "kind": "static", "n": 201, "shape": "polydisperse"},
        # a sweep of small collisions, bit-exact
        {"name": "batch_exact_256", "kind": "batch", "mode": "exact", "count": 256, "nt_hi": 200, "threads": 128,
         "steps": 20},
        # a sweep over the full range of sizes in the double-float form
        {"name": "batch_mixed_df_512", "kind": "batch", "mode": "mixed_df", "count": 512, "nt_hi": 1600,
         "threads": 512, "steps": 20},
        # the surrogate screens a sweep of a million points
        {"name": "predict_1m", "kind": "predict", "rows": 1000000},
        # loss and gradient of one batch
        {"name": "gradients_1024", "kind": "gradients", "rows": 1024},
        # one epoch over the training set of the study
        {"name": "train_45000", "kind": "train", "rows": 45000, "batch": 256},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["host_step", "loop", "loop", "loop", "static", "batch", "batch", "predict", "predict",
                       "gradients", "train"])
    mode = rng.choice(["exact", "exact", "mixed", "mixed_df"])
    shape = rng.choice(["cluster", "collision", "polydisperse"])
    if kind == "host_step":
        return {"kind": kind, "mode": mode, "n": _log_int(rng, 24, 5000), "shape": shape}
    if kind == "loop":
        n = _log_int(rng, 64, 20000)
        return {"kind": kind, "mode": mode, "n": n, "shape": shape, "skip": 100 if n <= 5000 else 20}
    if kind == "static":
        return {"kind": kind, "n": rng.randint(1, 256), "shape": rng.choice(["cluster", "polydisperse"])}
    if kind == "batch":
        if rng.random() < 0.5:
            return {"kind": kind, "mode": "exact", "count": _log_int(rng, 32, 512),
                    "nt_hi": _log_int(rng, 80, 300), "threads": rng.choice([64, 128, 256]), "steps": 20}
        return {"kind": kind, "mode": "mixed_df", "count": _log_int(rng, 32, 512), "nt_hi": _log_int(rng, 80, 1600),
                "threads": rng.choice([128, 256, 512]), "steps": 20}
    if kind == "predict":
        return {"kind": kind, "rows": _log_int(rng, 3, 1000000)}
    if kind == "gradients":
        return {"kind": kind, "rows": 32 * rng.randint(1, 32)}
    b = 32 * rng.choice([2, 4, 8, 16])
    return {"kind": kind, "rows": max(b, _log_int(rng, 512, 45000)), "batch": b}


# ------------------------------------------------------------------ inputs --
def _stir(g: BallGroup, rng, speed: float) -> None:
    """Squeezes the cluster and gives its spheres the relative motion and spin that a collision does: contacts
    slide and roll for many steps, instead of sticking at relative velocities near 0."""
    g.pos *= SQUEEZE
    g.vel += rng.normal(0.0, speed, g.vel.shape)
    g.w += rng.normal(0.0, speed / configs.RADIUS, g.w.shape)


def _group(case: dict, seed: int) -> tuple[BallGroup, float, float, float]:
    """A squeezed cluster or collision of case["n"] spheres and its dt, kin, kout."""
    n, shape, k_speed = case["n"], case["shape"], 1.0
    if shape == "collision":
        n_p = max(1, n // 5)
        g = configs.build_collision(n - n_p, n_p, 100.0, 1.0, 0.3, 2 * seed + 1, 2 * seed + 2)
        k_speed = 2.0
    elif shape == "polydisperse":
        g = configs.build_cluster(n, seed + 1, sigma_v=1e-2, sigma_ln=0.2)
    else:
        g = configs.build_cluster(n, seed + 1, sigma_v=1e-3)
    rng = np.random.default_rng([seed, n])
    _stir(g, rng, 4.0)
    kin, kout, dt = configs.spring_and_dt(float(g.R.max()), float(g.m.min()), k_speed)
    return g, dt, kin, kout


def _collisions(case: dict, seed: int, build: bool = True) -> list:
    """Collisions of the sweep's ranges: sizes by the case, clusters, speeds and materials by the seed."""
    cols = batch.sample_collisions(case["count"], 0, nt_range=(64, case["nt_hi"]), build=False)
    other = batch.sample_collisions(case["count"], seed + 1, build=False)
    for c, o in zip(cols, other):
        c.seed, c.speed, c.b_frac, c.cor, c.mu = o.seed, o.speed, o.b_frac, o.cor, o.mu
        if build:
            batch.build_instance(c)
            _stir(c.group, np.random.default_rng([seed, c.n]), 0.05 * c.speed)
    return cols


def _rows(case: dict, seed: int) -> tuple[np.ndarray, np.ndarray]:
    """Standardised features and smooth outcomes of them."""
    rng = np.random.default_rng([seed, case["rows"]])
    x = rng.standard_normal((case["rows"], NET["n_in"])).astype(np.float32)
    a = rng.standard_normal((NET["n_in"], NET["n_out"]))
    y = np.tanh(x @ a / 2) + 0.05 * rng.standard_normal((case["rows"], NET["n_out"]))
    return x, y.astype(np.float32)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    s = {"case": case}
    if kind in ("host_step", "loop"):
        g, dt, kin, kout = _group(case, seed)
        sim = GpuStep(g, configs.dust_material(), case["mode"])
        sim.set_scalars(dt, kin, kout)
        sim.init_conditions()
        sim.download()
        s["sim"] = sim
    elif kind == "static":
        g, _, kin, kout = _group(case, seed)
        dev = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")  # noqa: E731
        s["in"] = [dev(a) for a in (g.pos, g.vel, g.w, g.R, g.m, g.moi)]
        s["out"] = [dev(np.zeros_like(g.pos)), dev(np.zeros_like(g.pos)), dev(np.zeros(8))]
        s["mat"], s["k"], s["lib"] = configs.dust_material(), (kin, kout), _lib.lib()
    elif kind == "batch":
        run_ = batch.BatchRun(_collisions(case, seed), case["mode"], steps=case["steps"], skip=case["steps"])
        run_.set_shape(0, case["threads"])  # the pair-tile pass, which the autotuner picks at these sizes
        s["batch"] = run_
    else:
        s["x"], s["y"] = _rows(case, seed)
        s["net"] = Mlp(**NET, max_batch=max(1024, case.get("batch", 0)), seed=seed)
    return s


# -------------------------------------------------------------------- pass --
def _arrays(g: BallGroup) -> dict:
    return {k: getattr(g, k) for k in ("pos", "vel", "w", "acc", "aacc")}


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "host_step":
        state["sim"].sim_one_step_host(False)
        return _arrays(state["sim"].group)
    if kind == "loop":
        rows = state["sim"].sim_looper(case["skip"] + 1, case["skip"])
        out = _arrays(state["sim"].download())
        out["energy"] = np.array([[r.PE, r.KE, r.E, r.p, r.L] for r in rows])
        return out
    if kind == "static":
        ptr = [t.data_ptr() for t in state["in"]]
        acc, aacc, energy = state["out"]
        _lib.check(state["lib"].sl_forces_static(case["n"], *ptr, state["mat"], *state["k"], acc.data_ptr(),
                                                 aacc.data_ptr(), energy.data_ptr(),
                                                 torch.cuda.current_stream().cuda_stream), "sl_forces_static")
        return {"acc": acc, "aacc": aacc, "energy": energy}
    if kind == "batch":
        b = state["batch"]
        b.run(1, case["steps"], True)
        return {**b.state(), "energy": b.energy()}
    net = state["net"]
    if kind == "predict":
        return net.predict(state["x"])
    if kind == "gradients":
        loss, grads = net.gradients(state["x"], state["y"])
        return {"loss": np.float32(loss), "grads": grads}
    curve = net.train(state["x"], state["y"], epochs=1, batch=case["batch"], lr=1e-3, seed=1)
    return {"curve": curve, "params": net.params()}


# ------------------------------------------------------------------- work --
def work(case: dict) -> dict:
    kind = case["kind"]
    pair = 52.0  # flops of one pair out of contact (spacelab_gb300/flops.py)
    if kind in ("host_step", "loop"):
        n, steps = case["n"], case.get("skip", 1)
        return {"bytes": 2.0 * 5 * 24 * n, "flops": pair * n * (n - 1) / 2 * steps}
    if kind == "static":
        n = case["n"]
        return {"bytes": (3 * 24 + 3 * 8 + 2 * 24) * n + 64.0, "flops": pair * n * (n - 1) / 2 + 1}
    if kind == "batch":
        n = np.array([c.n for c in _collisions(case, 0, build=False)], dtype=np.float64)
        return {"bytes": float(2 * 5 * 24 * n.sum()),
                "flops": float(pair * (n * (n - 1) / 2).sum() * (case["steps"] + 1))}
    w = [NET["n_in"]] + [NET["hidden"]] * NET["layers"] + [NET["n_out"]]
    macs = float(sum(a * b for a, b in zip(w, w[1:])))
    params = macs + sum(w[1:])
    rows = case["rows"]
    io = 4.0 * rows * (NET["n_in"] + NET["n_out"])
    if kind == "predict":
        return {"bytes": io + 2 * params, "flops": 2 * macs * rows}
    if kind == "gradients":
        return {"bytes": io + 2 * params + 4 * params, "flops": 6 * macs * rows}
    return {"bytes": io + 8 * params, "flops": 6 * macs * rows}


# ----------------------------------------------- the same in plain 64 bits --
class _Systems:
    """Equal-length padded systems [I, n, 3] in FP64 and the reference step on them."""

    def __init__(self, groups, mats_us, dt, kin, kout, device):
        self.n = np.array([g.num_particles for g in groups])
        size = int(self.n.max())
        t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=device)  # noqa: E731

        def pad(name, fill):
            first = getattr(groups[0], name)
            out = np.full((len(groups), size) + first.shape[1:], fill)
            for i, g in enumerate(groups):
                out[i, : g.num_particles] = getattr(g, name)
            return t(out)

        self.pos, self.vel, self.w = pad("pos", 0.0), pad("vel", 0.0), pad("w", 0.0)
        self.R, self.m, self.moi = pad("R", 1.0), pad("m", 1.0), pad("moi", 1.0)
        self.live = torch.arange(size, device=device)[None, :] < torch.tensor(self.n, device=device)[:, None]
        self.dt, self.kin, self.kout, self.u_s = t(dt), t(kin), t(kout), t(mats_us)
        self.mat = configs.dust_material()
        self.prev = self.pos
        self.PE = torch.zeros(len(groups), dtype=torch.float64, device=device)
        self.acc = self.aacc = None

    def forces(self, energy: bool) -> None:
        inst, size = self.R.shape
        M = self.mat
        acc, aacc = torch.zeros_like(self.pos), torch.zeros_like(self.pos)
        pe = torch.zeros_like(self.PE)
        rows = max(1, min(size, int(4e7 // (inst * size))))
        touching = []
        for c0 in range(0, size, rows):
            c1 = min(size, c0 + rows)
            r = [self.pos[:, None, :, k] - self.pos[:, c0:c1, None, k] for k in range(3)]
            dist = (r[0] * r[0] + r[1] * r[1] + r[2] * r[2]).sqrt_()
            Ra, Rb = self.R[:, c0:c1, None], self.R[:, None, :]
            overlap = (Ra + Rb) - dist
            ok = self.live[:, c0:c1, None] & self.live[:, None, :]
            idx = torch.arange(c0, c1, device=ok.device)
            ok[:, torch.arange(c1 - c0, device=ok.device), idx] = False
            hit = ok & (overlap > 0)
            ok &= ~hit
            at = hit.nonzero()
            at[:, 1] += c0
            touching.append(at[at[:, 1] > at[:, 2]])
            h = overlap.abs_().clamp_(min=M.h_min)
            S = h * h + 2 * Ra * h + 2 * Rb * h
            T = S + 4 * Ra * Rb
            f = (M.Ha / 6 * 64 * Ra ** 3) * Rb ** 3 * ((h + Ra + Rb) / (S * S * T * T))
            f = torch.where(ok, f / dist, torch.zeros_like(f))
            for k in range(3):
                acc[:, c0:c1, k] = (f * r[k]).sum(-1) / self.m[:, c0:c1]
            if energy:
                u = -M.Ha / 6 * (2 * Ra * Rb / S + 2 * Ra * Rb / T + torch.log(S / T))
                pe += torch.where(ok, u, torch.zeros_like(u)).sum((1, 2)) / 2
        at = torch.cat(touching)
        if len(at):
            pe = pe + self._contacts(at, acc, aacc, energy)
        self.acc, self.aacc, self.PE = acc, aacc, pe

    def _contacts(self, at, acc, aacc, energy):
        I, A, B = at.unbind(1)
        M = self.mat
        norm = lambda v: v.norm(dim=-1)  # noqa: E731
        g = lambda a, k: a[I, k]  # noqa: E731
        r = g(self.pos, B) - g(self.pos, A)
        dist, old = norm(r), norm(g(self.prev, B) - g(self.prev, A))
        Ra, Rb, ma, mb = g(self.R, A), g(self.R, B), g(self.m, A), g(self.m, B)
        overlap = Ra + Rb - dist
        k = torch.where(dist >= old, self.kout[I], self.kin[I])
        n = r / dist[:, None]
        S = M.h_min ** 2 + 2 * (Ra + Rb) * M.h_min
        T = S + 4 * Ra * Rb
        coef = M.Ha / 6 * 64 * Ra ** 3 * Rb ** 3 * ((M.h_min + Ra + Rb) / (S * S * T * T))
        elastic = (-k * overlap / 2)[:, None] * n
        efm = norm(elastic)[:, None]
        ra, rb = r * (Ra / (Ra + Rb))[:, None], -r * (Rb / (Ra + Rb))[:, None]
        wa, wb = g(self.w, A), g(self.w, B)
        dv = g(self.vel, B) - g(self.vel, A)
        u = dv - (dv * r).sum(-1, keepdim=True) * r / (dist * dist)[:, None]
        u = u - torch.linalg.cross(wa, ra) - torch.linalg.cross(wb, ra)
        un, wd = norm(u)[:, None], wa - wb
        slide = torch.where(un > 1e-13, self.u_s[I][:, None] * efm * u / un, torch.zeros_like(u))
        c = torch.linalg.cross(wd, ra)
        roll = torch.where(norm(wd)[:, None] > 1e-13, -M.u_r * efm * c / norm(c)[:, None], torch.zeros_like(c))
        force = (M.G * ma * mb / (dist * dist))[:, None] * n + elastic + slide + coef[:, None] * n
        acc.index_put_((I, A), force / ma[:, None], accumulate=True)
        acc.index_put_((I, B), -force / mb[:, None], accumulate=True)
        aacc.index_put_((I, A), torch.linalg.cross(ra, slide + roll) / g(self.moi, A)[:, None], accumulate=True)
        aacc.index_put_((I, B), torch.linalg.cross(rb, roll - slide) / g(self.moi, B)[:, None], accumulate=True)
        pe = torch.zeros_like(self.PE)
        if energy:
            U = -M.Ha / 6 * (2 * Ra * Rb / S + 2 * Ra * Rb / T + torch.log(S / T)) + 0.5 * k * overlap * overlap
            pe.index_put_((I,), U, accumulate=True)
        return pe

    def step(self, energy: bool = False) -> None:
        dt = self.dt[:, None, None]
        velh, wh = self.vel + self.acc / 2 * dt, self.w + self.aacc / 2 * dt
        self.prev, self.pos = self.pos, self.pos + velh * dt
        self.forces(energy)
        self.vel, self.w = velh + self.acc / 2 * dt, wh + self.aacc / 2 * dt

    def totals(self) -> torch.Tensor:
        """[I, 8]: PE, KE, momentum, angular momentum."""
        live = self.live[..., None]
        m, moi = self.m[..., None], self.moi[..., None]
        ke = (0.5 * m * self.vel ** 2 + 0.5 * moi * self.w ** 2).where(live, torch.zeros_like(m)).sum((1, 2))
        mom = (m * self.vel).where(live, torch.zeros_like(m)).sum(1)
        L = (m * torch.linalg.cross(self.pos, self.vel) + moi * self.w).where(live, torch.zeros_like(m)).sum(1)
        return torch.cat([self.PE[:, None], ke[:, None], mom, L], 1)

    def arrays(self) -> dict:
        flat = lambda a: torch.cat([a[i, :k] for i, k in enumerate(self.n)]).cpu().numpy()  # noqa: E731
        return {k: flat(getattr(self, k)) for k in ("pos", "vel", "w", "acc", "aacc")}


def _network(p: np.ndarray, x, y, device):
    """(outputs, loss, gradient in the parameter vector's layout) of the network in FP64."""
    up = lambda v: (v + 31) // 32 * 32  # noqa: E731
    w = [NET["n_in"]] + [NET["hidden"]] * NET["layers"] + [NET["n_out"]]
    t = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=device)  # noqa: E731
    flat, layers, off = t(p), [], 0
    for a, b in zip(w, w[1:]):
        W = flat[off: off + up(a) * up(b)].reshape(up(b), up(a))[:b, :a].clone().requires_grad_(y is not None)
        off += up(a) * up(b)
        bias = flat[off: off + b].clone().requires_grad_(y is not None)
        off += up(b)
        layers.append((W, bias))
    v = t(x)
    for k, (W, bias) in enumerate(layers):
        v = v @ W.T + bias
        if k + 1 < len(layers):
            v = torch.nn.functional.gelu(v)
    if y is None:
        return v.cpu().numpy(), None, None
    loss = ((v - t(y)) ** 2).mean()
    loss.backward()
    grads = np.zeros(len(p))
    off = 0
    for (W, bias), a, b in zip(layers, w, w[1:]):
        part = np.zeros((up(b), up(a)))
        part[:b, :a] = W.grad.cpu().numpy()
        grads[off: off + part.size] = part.reshape(-1)
        off += part.size
        grads[off: off + b] = bias.grad.cpu().numpy()
        off += up(b)
    return None, float(loss), grads


def exact(case: dict, seed: int):
    kind = case["kind"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if kind in ("host_step", "loop", "static"):
        g, dt, kin, kout = _group(case, seed)
        s = _Systems([g], [configs.dust_material().u_s], [dt], [kin], [kout], device)
        s.forces(kind == "static")  # touching pairs start with k = kout: the previous positions are the current ones
        if kind == "static":
            return {"acc": s.acc[0], "aacc": s.aacc[0], "energy": s.totals()[0]}
        steps = case.get("skip", 1)
        for k in range(1, steps + 1):
            s.step(kind == "loop" and k == steps)
        out = s.arrays()
        if kind == "loop":
            e = s.totals()[0].cpu().numpy()
            out["energy"] = np.array([[e[0], e[1], e[0] + e[1], np.linalg.norm(e[2:5]), np.linalg.norm(e[5:8])]])
        return out
    if kind == "batch":
        cols = _collisions(case, seed)
        order = sorted(range(len(cols)), key=lambda i: cols[i].n)
        got, energy = [None] * len(cols), np.zeros((len(cols), 2, 8))
        at = 0
        while at < len(order):  # systems of like size together, padded to the largest of them
            end = at + 1
            while end < len(order) and cols[order[end]].n ** 2 * (end + 1 - at) <= 4e7:
                end += 1
            part = [cols[i] for i in order[at:end]]
            s = _Systems([c.group for c in part], [c.mu for c in part], [c.dt for c in part], [c.kin for c in part],
                         [c.kout for c in part], device)
            s.forces(True)
            energy[order[at:end], 0] = s.totals().cpu().numpy()
            for k in range(1, case["steps"] + 1):
                s.step(k == case["steps"])
            energy[order[at:end], 1] = s.totals().cpu().numpy()
            flat = s.arrays()
            cut = np.cumsum(s.n)[:-1]
            for name, a in flat.items():
                for i, piece in zip(order[at:end], np.split(a, cut)):
                    got[i] = got[i] or {}
                    got[i][name] = piece
            at = end
        out = {k: np.concatenate([p[k] for p in got]) for k in ("pos", "vel", "w", "acc", "aacc")}
        return {**out, "energy": energy}
    x, y = _rows(case, seed)
    if kind == "train":
        return None  # the rows of a batch follow the library's own shuffle
    p = Mlp(**NET, seed=seed).params()
    if kind == "predict":
        return _network(p, x, None, device)[0]
    _, loss, grads = _network(p, x, y, device)
    return {"loss": loss, "grads": grads}
