"""Workloads of the framework as a user's program runs them, for timing.

Every case is one pass of a loop that such a program runs many times, through
the public handles (Context, Batch, Network) and the C ABI behind them:

* ``loop``: a simulation between two observer outputs: `steps` steps, the
  order parameters (the observers' summary line) and the state, as a float
  trajectory frame in a page-locked buffer (GPU path) or as the FP64 state
  (reference arithmetic).  The reference's observers save every 10 steps
  (second order) or every 100 (first order).
* ``dropin``: one DoStep(system, state, t, dt) on a host state array, as a
  reference engine's time loop calls it.
* ``sweep``: a batch of independent systems run on between two order-parameter
  samples, with a checkpoint frame of all systems.
* ``train`` / ``predict``: the surrogate network fitted on run results, and
  evaluated over a phase-diagram grid.

``exact`` restates each of them in plain 64-bit torch from the equations and
the published methods (Philox4x32-10, Box-Muller, the steppers' schemes).
"""
import ctypes
import math

import numpy as np
import torch

import spsslangevinintegration_gb300 as spss
from spsslangevinintegration_gb300 import _native, sweep
from spsslangevinintegration_gb300.surrogate import Network

VARIANTS = {"dispatch": spss.VARIANT_DISPATCH, "all_pairs": spss.ALL_PAIRS, "linked_list": spss.LINKED_LIST,
            "linked_list_verlet": spss.LINKED_LIST_VERLET, "global_field": spss.GLOBAL_FIELD}
STEPPERS = {"rk4": spss.RK4, "se": spss.STOCHASTIC_EULER, "srk": spss.STOCHASTIC_RUNGE_KUTTA}
SKIN = 0.3
HIDDEN = 128


def listed():
    return [
        # The reference's plain deterministic run: first order, 1,000 particles at density 1, every pair, RK4 in
        # FP64, output every 100 steps.
        dict(name="rk4_f64_n1000", do="loop", model=1, precision="f64", variant="all_pairs", stepper="rk4", n=1000,
             density=1.0, dt=0.01, steps=100),
        # Reference arithmetic of the inertial model on its cell list (a validation run of the 65,536-particle
        # configuration), output every 10 steps.
        dict(name="list_f64_n65536", do="loop", model=2, precision="f64", variant="linked_list", stepper="se",
             n=65536, density=2.0, dt=0.005, steps=10),
        # Reference arithmetic of the first-order model as its engine dispatches it (linked list + Verlet), with the
        # order 1.5 stepper; an odd particle number.
        dict(name="verlet_f64_n20011", do="loop", model=1, precision="f64", variant="linked_list_verlet",
             stepper="srk", n=20011, density=2.0, dt=0.005, steps=10),
        # The ordinary inertial run: 65,536 particles, cell list rebuilt every step, Euler-Maruyama.
        dict(name="cells_f32_n65536", do="loop", model=2, precision="f32", variant="linked_list", stepper="se",
             n=65536, density=2.0, dt=0.005, steps=10),
        # The large single system: 4,194,304 particles, Verlet lists with skin 0.3 R, order 1.5 stepper.
        dict(name="verlet_f32_n4194304", do="loop", model=2, precision="f32", variant="linked_list_verlet",
             stepper="srk", n=4194304, density=2.0, dt=0.005, steps=10),
        # First-order model in its own polar order field (a parameter continuation's setting, on the GPU path).
        dict(name="global_f32_n999983", do="loop", model=1, precision="f32", variant="global_field", stepper="srk",
             n=999983, density=1.0, dt=0.005, steps=100),
        # A wide interaction radius: the dispatch evaluates every pair (radius 0.3 of the box).
        dict(name="allpairs_f32_n4000", do="loop", model=2, precision="f32", variant="dispatch", stepper="se",
             n=4000, density=0.0, dt=0.005, steps=10),
        # A small reference engine switched over to the drop-in classes: one DoStep on the host array.
        dict(name="dropin_f32_n2000", do="dropin", model=1, precision="f32", variant="linked_list_verlet",
             stepper="srk", n=2000, density=2.0, dt=0.005, steps=1),
        # The phase-diagram sweep: 512 systems of 1,024 to 65,536 particles (log-uniform), cell lists.
        dict(name="sweep_cells_512", do="sweep", variant="linked_list", systems=512, n_min=1024, n_max=65536,
             dt=0.005, steps=10),
        # Training runs of the surrogate: many small systems of one size on per-system Verlet lists.
        dict(name="sweep_verlet_1024x1024", do="sweep", variant="linked_list_verlet", systems=1024, n_min=1024,
             n_max=1024, dt=0.005, steps=20),
        # One epoch of fitting the surrogate on a set of run results.
        dict(name="train_16384", do="train", n=16384, batch=1024, epochs=1),
        # The surrogate over a 256 x 256 phase-diagram grid.
        dict(name="predict_65536", do="predict", n=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("f64", "f64", "cells", "verlet", "global", "allpairs", "dropin", "sweep", "sweep", "train",
                       "predict"))
    model = rng.choice((1, 2))
    if kind == "f64":
        variant = rng.choice(("all_pairs", "linked_list", "linked_list_verlet"))
        stepper = rng.choice(("rk4", "se", "srk"))
        n = _log_int(rng, 500, 5000) if variant == "all_pairs" else _log_int(rng, 1000, 80000)
        return dict(do="loop", model=model, precision="f64", variant=variant, stepper=stepper, n=n,
                    density=rng.choice((1.0, 2.0)), dt=0.005, steps=10)
    if kind in ("cells", "verlet"):
        big = 4000000 if kind == "verlet" else 2000000
        return dict(do="loop", model=model, precision="f32",
                    variant="linked_list" if kind == "cells" else "linked_list_verlet",
                    stepper=rng.choice(("se", "srk")), n=_log_int(rng, 1000, big), density=rng.choice((1.0, 2.0)),
                    dt=0.005, steps=10)
    if kind == "global":
        return dict(do="loop", model=1, precision="f32", variant="global_field", stepper=rng.choice(("se", "srk")),
                    n=_log_int(rng, 1000, 1000000), density=1.0, dt=0.005, steps=rng.choice((10, 100)))
    if kind == "allpairs":
        return dict(do="loop", model=2, precision="f32", variant="dispatch", stepper=rng.choice(("se", "srk")),
                    n=_log_int(rng, 200, 12000), density=0.0, dt=0.005, steps=10)
    if kind == "dropin":
        return dict(do="dropin", model=model, precision="f32",
                    variant=rng.choice(("linked_list", "linked_list_verlet")), stepper=rng.choice(("se", "srk")),
                    n=_log_int(rng, 1000, 500000), density=2.0, dt=0.005, steps=1)
    if kind == "sweep":
        if rng.random() < 0.5:
            n = _log_int(rng, 700, 3000)
            return dict(do="sweep", variant=rng.choice(("linked_list", "linked_list_verlet")),
                        systems=_log_int(rng, 64, 1024), n_min=n, n_max=n, dt=0.005, steps=20)
        return dict(do="sweep", variant=rng.choice(("linked_list", "linked_list_verlet")),
                    systems=_log_int(rng, 16, 300), n_min=1024, n_max=_log_int(rng, 4096, 65536), dt=0.005, steps=10)
    if kind == "train":
        return dict(do="train", n=_log_int(rng, 4096, 50000), batch=rng.choice((512, 1024, 2048)), epochs=1)
    return dict(do="predict", n=_log_int(rng, 100, 65536))


# ---------------------------------------------------------------- inputs


def _single_params(case, seed):
    """make_params keywords of a single system, mapped to the unit box (sweep.py)."""
    n, model = case["n"], case["model"]
    if case["density"] > 0.0:
        L = math.sqrt(n / case["density"])
        rho = 1.0 / L
    else:
        L, rho = 1.0, 0.3
    kw = dict(model=model, n=n, rho=rho, seed=seed & 0xFFFFFFFF,
              precision=spss.PRECISION_F64 if case["precision"] == "f64" else spss.PRECISION_F32,
              variant=VARIANTS[case["variant"]])
    if model == 1:
        kw.update(v0=0.1 / L, xi=0.1, sigma=1.0, D_phi=0.1)
    else:
        kw.update(v0=0.5 / L, xi_r=1.0, xi_phi=1.0, sigma=1.0, D_phi=0.1)
    if case["variant"] == "linked_list_verlet":
        kw["r_max"] = rho * (1.0 + SKIN)
        kw["nc_verlet"] = int(1.0 / kw["r_max"])
    return kw, L


def _single_state(case, L, seed):
    """Uniform positions and phases; second order: a unit velocity along the phase; omega = 0."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    if case["model"] == 2:
        return sweep.initial_state(n, L, seed)
    x = np.zeros((n, 4))
    x[:, 0], x[:, 1] = rng.random(n), rng.random(n)
    x[:, 2] = rng.uniform(-np.pi, np.pi, n)
    return x.reshape(-1)


def _frequencies(case, seed):
    return np.random.default_rng(seed + 17).normal(0.0, 0.5, case["n"])


def _sweep_points(case, seed):
    """Seeded parameter points; the sizes are the case's own."""
    span = (case["n_min"], case["n_max"] + 0.5)
    sizes = sweep.replica_table(case["systems"], seed=0, n_range=span)
    points = sweep.replica_table(case["systems"], seed=seed, n_range=span)
    return [dict(p, n=q["n"]) for p, q in zip(points, sizes)]


def _data(case, seed):
    """Standardised parameter points and smooth order-parameter surfaces over them, with run-to-run noise."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1.7, 1.7, (case["n"], 5)).astype(np.float32)
    s = 1.0 / (1.0 + np.exp(-2.0 * (x[:, 0] - 0.8 * x[:, 1])))
    t = np.stack([s, s * s, 0.3 * s * (1.0 - s), 0.2 * (1.0 - s)], axis=1)
    t = (t + rng.normal(0.0, 0.1, t.shape)).astype(np.float32)
    return x, t


def _weights(seed):
    """A network's flat parameters, uniform in +-1/sqrt(fan_in), zero biases."""
    rng = np.random.default_rng(seed + 29)
    parts = []
    for out, fan in ((HIDDEN, 5), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (4, HIDDEN)):
        parts += [rng.uniform(-1.0, 1.0, out * fan) / math.sqrt(fan), np.zeros(out)]
    return np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    seed = int(seed)
    do = case["do"]
    if do in ("train", "predict"):
        net = Network(seed)
        net.params = _weights(seed)
        x, t = _data(case, seed)
        if do == "train":
            net.set_data(x, t)
        return dict(case=case, net=net, x=x, seed=seed)
    if do == "sweep":
        skin = SKIN if case["variant"] == "linked_list_verlet" else 0.0
        ctx = sweep.make_batch(_sweep_points(case, seed), variant=VARIANTS[case["variant"]], seed=seed & 0xFFFFFFFF,
                               skin=skin, state_seed=seed % 1000)
        return dict(case=case, ctx=ctx, frame=spss.PinnedArray(ctx.length, np.float32))
    kw, L = _single_params(case, seed)
    ctx = spss.Context(kw.pop("model"), kw.pop("n"), kw.pop("rho"), **kw)
    state = _single_state(case, L, seed)
    if do == "dropin":
        host = spss.PinnedArray(ctx.length)
        host.array[:] = state
        return dict(case=case, ctx=ctx, host=host, t=0.0)
    if case["variant"] == "global_field":
        ctx.set_natural_frequencies(_frequencies(case, seed))
    ctx.set_state(state)
    frame = spss.PinnedArray(ctx.length, np.float32) if case["precision"] == "f32" else None
    return dict(case=case, ctx=ctx, frame=frame, t=0.0)


# ---------------------------------------------------------------- one pass


def _frame(ctx, buf):
    """The state as a float trajectory frame in the page-locked buffer (what observers.TrajectoryWriter queues)."""
    a = buf.array
    _native.check(ctx.L.spss_frame_async(ctx.h, _native.FRAME_RAW, a.ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                                         a.size), "spss_frame_async")
    ctx.synchronize()
    return a


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "train":
        net = state["net"]
        loss = net.train(case["epochs"], batch=case["batch"], lr=2e-3, seed=state["seed"])
        return {"loss": loss, "params": net.params}
    if do == "predict":
        return {"y": state["net"].forward(state["x"])}
    ctx = state["ctx"]
    if do == "sweep":
        ctx.run(spss.STOCHASTIC_EULER, 0.0, case["dt"], case["steps"], sample_every=10, sample_from=1)
        return {"stats": ctx.stats(), "order": ctx.system_order_parameters(), "frame": _frame(ctx, state["frame"])}
    stepper = STEPPERS[case["stepper"]]
    t, dt = state["t"], case["dt"]
    state["t"] = t + case["steps"] * dt
    if do == "dropin":
        return {"state": ctx.step_host(stepper, state["host"].array, t, dt)}
    ctx.steps(stepper, t, dt, case["steps"])
    order = ctx.order_parameters()
    if state["frame"] is not None:
        return {"order": order, "frame": _frame(ctx, state["frame"])}
    return {"order": order, "state": ctx.get_state()}


# ---------------------------------------------------------------- work


def _neighbours(case):
    """Mean number of neighbours within R."""
    if case["variant"] == "dispatch":
        return math.pi * 0.3 * 0.3 * case["n"]
    return math.pi * case.get("density", 2.0)


def work(case):
    do = case["do"]
    if do in ("train", "predict"):
        macs = 5 * HIDDEN + 2 * HIDDEN * HIDDEN + HIDDEN * 4
        params = macs + 3 * HIDDEN + 4
        if do == "predict":
            return {"bytes": 4.0 * case["n"] * 9 + 4.0 * params, "flops": 2.0 * macs * case["n"]}
        back = 3 * macs - 5 * HIDDEN  # forward, dZ chain (not to the inputs), weight gradients
        updates = -(-case["n"] // case["batch"])
        return {"bytes": case["epochs"] * (4.0 * case["n"] * 9 + 24.0 * params * updates),
                "flops": 2.0 * back * case["n"] * case["epochs"]}
    if do == "sweep":
        n = sum(p["n"] for p in _sweep_points(case, 0))
        model, word = 2, 4
    else:
        n, model, word = case["n"], case["model"], 8 if case["precision"] == "f64" else 4
    s = 4 if model == 1 else 6
    evals = 4 if case.get("stepper") == "rk4" else 1
    pair = 0.0 if case["variant"] == "global_field" else 12.0 * _neighbours(case)
    if case["variant"] in ("all_pairs", "dispatch"):
        pair += 5.0 * n
    # the state read and written once a step (positions at least 8 bytes), then once more for the output
    per_step = 2.0 * (2 * 8 + (s - 2) * word) * evals
    out = s * 8.0 * 2 if do == "dropin" else s * (8.0 if word == 8 else 4.0)
    return {"bytes": n * (per_step * case["steps"] + out), "flops": n * case["steps"] * evals * (pair + 60.0)}


# ---------------------------------------------------------------- 64-bit restatement


def _mul32(a, b):
    """High and low words of the product of 32-bit words held in int64 tensors."""
    p0 = (a & 0xFFFF) * b
    p1 = (a >> 16) * b
    low = p0 + ((p1 & 0xFFFF) << 16)
    return (p1 >> 16) + (low >> 32), low & 0xFFFFFFFF


def _philox(particle, replica, step, seed, block):
    """Philox4x32-10 (Salmon et al., SC'11), counter (particle, step lo, step hi, replica << 8 | block)."""
    c0 = particle
    c1 = torch.full_like(particle, step & 0xFFFFFFFF)
    c2 = torch.full_like(particle, step >> 32)
    c3 = ((replica << 8) | block) & 0xFFFFFFFF
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    m0, m1 = 0xD2511F53, 0xCD9E8D57
    for _ in range(10):
        h0, l0 = _mul32(c0, torch.full_like(c0, m0))
        h1, l1 = _mul32(c2, torch.full_like(c2, m1))
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _pair(u1, angle):
    r = torch.sqrt(-2.0 * torch.log(u1))
    return r * torch.cos(angle), r * torch.sin(angle)


def _normals(f64, need, particle, replica, step, seed):
    """The standard normals of one step (list of `need` tensors), from the Philox words by Box-Muller: 32-bit
    uniforms (FP64 path), 24-bit uniforms, or three pairs with 16-bit angles from one block (GPU path)."""
    u = _philox(particle, replica, step, seed, 0)
    if f64:
        if need > 4:
            u = u + _philox(particle, replica, step, seed, 1)
        z = []
        for a, b in zip(u[::2], u[1::2]):
            z += _pair((a.double() + 0.5) * 2.0 ** -32, 2.0 * math.pi * (b.double() + 0.5) * 2.0 ** -32)
        return z[:need]
    z = []
    if need > 4:
        angles = (u[3] & 0xFFFF, u[3] >> 16, (u[0] & 0xFF) | ((u[1] & 0xFF) << 8))
        for a, b in zip(u[:3], angles):
            z += _pair(((a >> 8).double() + 0.5) * 2.0 ** -24, 2.0 * math.pi * ((b.double() + 0.5) * 2.0 ** -16 - 0.5))
    else:
        for a, b in zip(u[::2], u[1::2]):
            z += _pair(((a >> 8).double() + 0.5) * 2.0 ** -24, 2.0 * math.pi * ((b >> 8).double() * 2.0 ** -24 - 0.49999997))
    return z[:need]


class _Exact:
    """The particle systems of a case (one, or a batch) in FP64, their state as columns."""

    def __init__(self, systems, states, f64, frequencies=None):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.model = systems[0]["model"]
        s = 4 if self.model == 1 else 6
        x = torch.from_numpy(np.concatenate(states)).to(dev).reshape(-1, s).double()
        cols = [c.contiguous() for c in x.T]
        self.px, self.py, self.phi, self.w = cols[0], cols[1], cols[-2], cols[-1]
        self.vx, self.vy = (cols[2], cols[3]) if self.model == 2 else (None, None)
        sizes = torch.tensor([p["n"] for p in systems], device=dev)
        self.sizes = [p["n"] for p in systems]
        self.sys = torch.repeat_interleave(torch.arange(len(systems), device=dev), sizes)
        self.first = torch.cumsum(sizes, 0) - sizes
        self.local = torch.arange(x.shape[0], device=dev) - self.first[self.sys]
        self.replica = torch.tensor([p.get("replica", 0) for p in systems], device=dev)[self.sys]
        col = lambda key: torch.tensor([float(p.get(key, 0.0)) for p in systems], dtype=torch.float64, device=dev)[self.sys]  # noqa: E731
        self.v0, self.sigma, self.rho2 = col("v0"), col("sigma"), col("rho") ** 2
        self.xi_r = col("xi_r")
        self.xi_w = col("xi") if self.model == 1 else col("xi_phi")
        self.b_r, self.b_w = torch.sqrt(2.0 * col("D_r")), torch.sqrt(2.0 * col("D_phi"))
        self.systems, self.f64, self.seed = systems, f64, systems[0]["seed"]
        self.nu = None if frequencies is None else torch.from_numpy(frequencies).to(dev)
        nc = [max(1, int(1.0 / p["rho"])) for p in systems]
        self.dense = min(nc) < 16  # few cells: every pair is tested
        t = torch.tensor(nc, device=dev)
        self.nc = t[self.sys]
        self.cell0 = (torch.cumsum(t * t, 0) - t * t)[self.sys]
        self.ncell = int((t * t).sum())
        self.kept = {}

    def _sums(self, px, py, phi, w):
        """Per particle: neighbours within R, sum sin(phi_j - phi_i), sum (w_j - w_i) cos(phi_j - phi_i)."""
        n = px.numel()
        if self.dense or n <= 1500:
            card, torque, comp = [], [], []
            rows = max(1, 20000000 // n)
            for a in range(0, n, rows):
                b = min(n, a + rows)
                dx, dy = px[None, :] - px[a:b, None], py[None, :] - py[a:b, None]
                dx, dy = dx - torch.round(dx), dy - torch.round(dy)
                near = (dx * dx + dy * dy <= self.rho2[a:b, None]) & (self.sys[None, :] == self.sys[a:b, None])
                near[torch.arange(b - a), torch.arange(a, b)] = False
                d = phi[None, :] - phi[a:b, None]
                card.append(near.sum(1).double())
                torque.append(torch.where(near, torch.sin(d), 0.0).sum(1))
                comp.append(torch.where(near, (w[None, :] - w[a:b, None]) * torch.cos(d), 0.0).sum(1))
            return torch.cat(card), torch.cat(torque), torch.cat(comp)
        fx, fy = px - torch.floor(px), py - torch.floor(py)
        top = self.nc - 1
        cx = torch.minimum((fx * self.nc).long(), top)
        cy = torch.minimum((fy * self.nc).long(), top)
        cell = self.cell0 + cy * self.nc + cx
        order = torch.argsort(cell)
        count = torch.bincount(cell, minlength=self.ncell)
        start = torch.cumsum(count, 0) - count
        sx, sy, sp, sw = fx[order], fy[order], phi[order], w[order]
        ox, oy, nc, cell0, rho2 = cx[order], cy[order], self.nc[order], self.cell0[order], self.rho2[order]
        card, torque, comp = (torch.zeros(n, dtype=torch.float64, device=px.device) for _ in range(3))
        for ddy in (-1, 0, 1):
            for ddx in (-1, 0, 1):
                c = cell0 + torch.remainder(oy + ddy, nc) * nc + torch.remainder(ox + ddx, nc)
                i = torch.arange(n, device=px.device)
                b, k = start[c], count[c]
                m = 0
                while i.numel():
                    live = k > m
                    i, b, k = i[live], b[live], k[live]
                    j = b + m
                    dx, dy = sx[j] - sx[i], sy[j] - sy[i]
                    dx, dy = dx - torch.round(dx), dy - torch.round(dy)
                    near = (dx * dx + dy * dy <= rho2[i]) & (i != j)
                    a, q = i[near], j[near]
                    d = sp[q] - sp[a]
                    card[a] += 1.0
                    torque[a] += torch.sin(d)
                    comp[a] += (sw[q] - sw[a]) * torch.cos(d)
                    m += 1
        out = []
        for v in (card, torque, comp):
            r = torch.empty_like(v)
            r[order] = v
            out.append(r)
        return out

    def torque(self, px, py, phi, w, keep=None):
        """Torque derivative and complementary force.  A particle without neighbours has derivative 0, or (RK4)
        what the same stage of the step before left there."""
        if self.nu is not None:
            z = torch.polar(torch.ones_like(phi), phi)
            zm, wm = z.mean(), (w * z).mean()
            f = -self.xi_w * w + self.nu + self.sigma * zm.abs() * torch.sin(zm.angle() - phi)
            c = self.sigma * (wm.abs() * torch.cos(wm.angle() - phi) - w * zm.abs() * torch.cos(zm.angle() - phi))
            return f, c
        card, torque, comp = self._sums(px, py, phi, w)
        some = card > 0
        card = torch.clamp(card, min=1.0)
        old = self.kept.get(keep, torch.zeros_like(w)) if keep is not None else torch.zeros_like(w)
        f = torch.where(some, -self.xi_w * w + self.sigma * torque / card, old)
        if keep is not None:
            self.kept[keep] = f
        return f, torch.where(some, self.sigma * comp / card, torch.zeros_like(w))

    def _rhs(self, y, keep):
        px, py, vx, vy, phi, w = y
        f, _ = self.torque(px, py, phi, w, keep)
        c, s = torch.cos(phi), torch.sin(phi)
        if self.model == 1:
            return (self.v0 * c, self.v0 * s, None, None, w, f)
        return vx, vy, -self.xi_r * vx + self.v0 * c, -self.xi_r * vy + self.v0 * s, w, f

    def step(self, stepper, dt, index):
        y = (self.px, self.py, self.vx, self.vy, self.phi, self.w)
        if stepper == "rk4":
            add = lambda k, h: tuple(None if a is None else a + h * b for a, b in zip(y, k))  # noqa: E731
            k1 = self._rhs(y, 0)
            k2 = self._rhs(add(k1, 0.5 * dt), 1)
            k3 = self._rhs(add(k2, 0.5 * dt), 2)
            k4 = self._rhs(add(k3, dt), 3)
            y = tuple(None if a is None else a + (p + 2.0 * q + 2.0 * r + u) * dt / 6.0
                      for a, p, q, r, u in zip(y, k1, k2, k3, k4))
            self.px, self.py, self.vx, self.vy, self.phi, self.w = y
            return
        srk = stepper == "srk"
        need = (2 if srk else 1) if self.model == 1 else (6 if srk else 3)
        z = _normals(self.f64, need, self.local, self.replica, index, self.seed)
        f, comp = self.torque(self.px, self.py, self.phi, self.w)
        c, s, w = torch.cos(self.phi), torch.sin(self.phi), self.w
        sq, h2 = math.sqrt(dt), 0.5 * dt * dt
        wiener = lambda a, b: (a * sq, 0.5 * dt ** 1.5 * (a + b / math.sqrt(3.0)))  # noqa: E731
        if self.model == 1:
            fx, fy = self.v0 * c, self.v0 * s
            if srk:
                dw_, dz_ = wiener(z[0], z[1])
                self.px, self.py = self.px + fx * dt - w * fy * h2, self.py + fy * dt + w * fx * h2
                self.phi = self.phi + w * dt + f * h2 + self.b_w * dz_
                self.w = w + f * dt + (comp - self.xi_w * f) * h2 + self.b_w * (dw_ - self.xi_w * dz_)
            else:
                self.px, self.py, self.phi = self.px + fx * dt, self.py + fy * dt, self.phi + w * dt
                self.w = w + f * dt + self.b_w * sq * z[0]
            return
        ax, ay = -self.xi_r * self.vx + self.v0 * c, -self.xi_r * self.vy + self.v0 * s
        vx, vy = self.vx, self.vy
        if srk:
            (wx, zx), (wy, zy), (ww, zw) = wiener(z[0], z[1]), wiener(z[2], z[3]), wiener(z[4], z[5])
            self.px, self.py = self.px + vx * dt + ax * h2 + self.b_r * zx, self.py + vy * dt + ay * h2 + self.b_r * zy
            self.vx = vx + ax * dt + (-self.xi_r * ax - self.v0 * s * w) * h2 + self.b_r * (wx - self.xi_r * zx)
            self.vy = vy + ay * dt + (-self.xi_r * ay + self.v0 * c * w) * h2 + self.b_r * (wy - self.xi_r * zy)
            self.phi = self.phi + w * dt + f * h2 + self.b_w * zw
            self.w = w + f * dt + (comp - self.xi_w * f) * h2 + self.b_w * (ww - self.xi_w * zw)
        else:
            self.px, self.py, self.phi = self.px + dt * vx, self.py + dt * vy, self.phi + dt * w
            self.vx, self.vy = vx + dt * ax + sq * self.b_r * z[0], vy + dt * ay + sq * self.b_r * z[1]
            self.w = w + dt * f + sq * self.b_w * z[2]

    def order(self):
        """(R, arg R, R_v, arg R_v) of every system."""
        def per_system(re, im):
            k = len(self.sizes)
            sums = [torch.zeros(k, dtype=torch.float64, device=re.device).index_add_(0, self.sys, v) for v in (re, im)]
            z = torch.complex(sums[0], sums[1]) / torch.tensor(self.sizes, device=re.device)
            return z.abs(), z.angle()

        a = per_system(torch.cos(self.phi), torch.sin(self.phi))
        if self.model == 1:
            b = a
        else:
            v = torch.hypot(self.vx, self.vy)
            v = torch.where(v > 0, v, torch.full_like(v, math.inf))
            b = per_system(self.vx / v, self.vy / v)
        return torch.stack([a[0], a[1], b[0], b[1]], dim=1).cpu().numpy()

    def state(self):
        cols = [self.px, self.py] + ([self.vx, self.vy] if self.model == 2 else []) + [self.phi, self.w]
        return torch.stack(cols, dim=1).reshape(-1).cpu().numpy()


def _exact_network(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, t = (torch.from_numpy(v).to(dev).double() for v in _data(case, seed))
    flat = torch.from_numpy(_weights(seed)).to(dev).double()

    def forward(p, x):
        o = 0
        for out, fan, last in ((HIDDEN, 5, 0), (HIDDEN, HIDDEN, 0), (HIDDEN, HIDDEN, 0), (4, HIDDEN, 1)):
            W, b = p[o:o + out * fan].reshape(out, fan), p[o + out * fan:o + out * fan + out]
            o += out * fan + out
            x = x @ W.T + b
            if not last:
                x = torch.nn.functional.gelu(x)
        return x

    return {"y": forward(flat, x).cpu().numpy()}


def exact(case, seed):
    seed = int(seed)
    do = case["do"]
    if do == "train":
        return None  # the order of the minibatches is the library's own
    if do == "predict":
        return _exact_network(case, seed)
    if do == "sweep":
        points = _sweep_points(case, seed)
        if sum(p["n"] for p in points) * case["steps"] > 100000000:
            return None
        skin = SKIN if case["variant"] == "linked_list_verlet" else 0.0
        systems = [sweep.system_params(p, variant=VARIANTS[case["variant"]], seed=seed & 0xFFFFFFFF, replica=i,
                                       skin=skin) for i, p in enumerate(points)]
        states = [sweep.initial_state(p["n"], np.sqrt(p["n"] / p["density"]), (seed % 1000) * 1000003 + i)
                  for i, p in enumerate(points)]
        E = _Exact(systems, states, False)
        samples = []
        for k in range(case["steps"]):
            E.step("se", case["dt"], k)
            if (k + 1) % 10 == 0:
                samples.append(E.order())
        a = np.stack(samples)[:, :, [0, 2]]
        mean, var = a.mean(axis=0), a.var(axis=0)
        count = np.full(len(points), float(len(samples)))
        stats = np.stack([mean[:, 0], var[:, 0], mean[:, 1], var[:, 1], count], axis=1)
        return {"stats": stats, "order": E.order(), "frame": E.state()}
    kw, L = _single_params(case, seed)
    f64 = case["precision"] == "f64"
    freq = _frequencies(case, seed) if case["variant"] == "global_field" else None
    E = _Exact([kw], [_single_state(case, L, seed)], f64, freq)
    for k in range(case["steps"]):
        E.step(case["stepper"], case["dt"], k)
    if do == "dropin":
        return {"state": E.state()}
    return {"order": E.order()[0], "state" if f64 else "frame": E.state()}
