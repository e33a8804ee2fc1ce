"""Performance cases: the calls a simulation program makes, over the range of sizes it makes them at.

Disks are Keplerian (surface density r^-1.5, Rayleigh eccentricity and
inclination) around a unit-mass star, as the configurations of the benchmark
draw them; every case makes its own from the seed, on the GPU.  Kinds:

* ``step``: ``Sim.step`` with the state then read into device tensors (the
  loop of a run between two looks at the state);
* ``ensemble``: ``Ensemble.step`` and the same read-out, disks of uneven size;
* ``gradient``: a trajectory through ``disk_trajectory``, its eccentricity
  loss and the gradient of it;
* ``phases``: one step through the launchers of the phase interface, in the
  order of the reference's main loop;
* ``fof``: friends-of-friends groups of one snapshot;
* ``direct``: FP64 direct-sum forces on sampled targets (the error study);
* ``host``: ``Sim.step_host``, the state in pinned host memory on both sides.

``exact`` is the same arithmetic in FP64 with direct-sum self-gravity, in
plain torch.
"""
import importlib
import math

import numpy as np
import torch

nb = importlib.import_module("nbody-sim_b200")

KEYS = ("x", "y", "z", "vx", "vy", "vz")
ACC = ("ax", "ay", "az")
MJUP = float(np.float32(9.5479e-4))  # solar masses, include/Config.h of the reference
STATES = {"f32": nb.STATE_F32, "f64": nb.STATE_F64, "f32x2": nb.STATE_F32X2}


# ------------------------------------------------------------------ cases
def _step(name, n, state, steps, **kw):
    c = {"name": name, "kind": "step", "n": n, "state": state, "steps": steps, "mass": 1e-8,
         "r_min": 0.5, "r_max": 5.0, "eps": 1e-3, "theta": 0.5, "dt": 0.005, "r_coll": 0.0,
         "drag": 0.0, "pert_mass": 0.0, "pert_radius": 5.2}
    c.update(kw)
    return c


def listed():
    return [
        # the small disk: ten steps between two outputs, collisions on
        _step("step_4096", 4096, "f32", 10, dt=0.01, r_coll=7.790107e-6),
        # an ordinary disk of no special size, hi/lo state, gas and a planet
        _step("step_30011_hilo", 30011, "f32x2", 10, drag=1e-3, pert_mass=3.0, pert_radius=10.0,
              theta=0.7),
        # the full-physics run: FP64 state, collisions, gas, a planet
        _step("step_131072_full", 131072, "f64", 10, r_coll=3.8950534e-5, drag=1e-3,
              pert_mass=1.0),
        # the headline: a million bodies, gravity only
        _step("step_1048576", 1048576, "f32", 4, mass=1e-9, r_min=0.3, r_max=30.0, eps=5e-4,
              dt=0.002),
        # the largest: four times the headline
        _step("step_4194304", 4194304, "f32", 2, mass=1e-9, r_min=0.3, r_max=30.0, eps=5e-4,
              dt=0.002),
        # a sweep over perturbers: 64 disks of uneven size at once
        {"name": "ensemble_64", "kind": "ensemble", "disks": 64, "n_lo": 2048, "n_hi": 65536,
         "layout": 0, "steps": 4, "r_coll": 3.8950534e-5, "drag": 1e-3},
        # gradient of a final-state loss, every level kept
        {"name": "gradient_65536", "kind": "gradient", "n": 65536, "steps": 20, "mode": "tape",
         "every": 0},
        # the same with checkpoints and levels rebuilt backwards
        {"name": "gradient_20011_ckpt", "kind": "gradient", "n": 20011, "steps": 20,
         "mode": "checkpoint", "every": 5},
        # one step through the launchers, as a program written for the reference calls them
        {"name": "phases_100003", "kind": "phases", "n": 100003, "r_coll": 3.8950534e-5,
         "drag": 1e-3, "pert_mass": 1.0, "pert_radius": 5.2},
        # groups of a snapshot of the full-physics run
        {"name": "fof_131072", "kind": "fof", "n": 131072, "link": 2e-3},
        # the error study: sampled targets against every body
        {"name": "direct_1048576", "kind": "direct", "n": 1048576, "targets": 16384,
         "phi": False},
        # a step with the state coming from and going to host memory
        {"name": "host_1048576", "kind": "host", "n": 1048576},
    ]


def _log_int(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n + rng.randrange(2)))


def draw(rng):
    """One more case of the same kinds: any size in the range, options mixed."""
    kind = rng.choice(["step"] * 4 + ["ensemble", "gradient", "phases", "fof", "direct", "host"])
    if kind == "step":
        n = _log_int(rng, 1024, 4194304)
        big = n > 500000
        rc = 0.0 if big else rng.choice([0.0, 7.790107e-6, 3.8950534e-5])
        kw = {"r_coll": rc, "drag": rng.choice([0.0, 1e-3]),
              "pert_mass": rng.choice([0.0, 1.0, 3.0]),
              "theta": 0.5 if big else rng.choice([0.3, 0.5, 0.7]),
              "state": rng.choice(["f32", "f64", "f32x2"]),
              "steps": max(1, min(10, 4194304 // n))}
        if big:
            kw.update(mass=1e-9, r_min=0.3, r_max=30.0, eps=5e-4, dt=0.002)
        c = _step("", n, kw.pop("state"), kw.pop("steps"), **kw)
        del c["name"]
        return c
    if kind == "ensemble":
        return {"kind": kind, "disks": rng.randrange(2, 97), "n_lo": rng.choice([1024, 2048]),
                "n_hi": rng.choice([8192, 16384, 65536]), "layout": rng.randrange(1000),
                "steps": rng.randrange(1, 5), "r_coll": rng.choice([0.0, 3.8950534e-5]),
                "drag": rng.choice([0.0, 1e-3])}
    if kind == "gradient":
        n = _log_int(rng, 1024, 131072)
        mode = rng.choice(["tape", "checkpoint"])
        return {"kind": kind, "n": n, "steps": rng.randrange(8, 21), "mode": mode,
                "every": 0 if mode == "tape" else rng.randrange(3, 9)}
    if kind == "phases":
        return {"kind": kind, "n": _log_int(rng, 1024, 1000000),
                "r_coll": rng.choice([0.0, 3.8950534e-5]), "drag": rng.choice([0.0, 1e-3]),
                "pert_mass": rng.choice([0.0, 1.0]), "pert_radius": 5.2}
    if kind == "fof":
        n = _log_int(rng, 1024, 1000000)
        return {"kind": kind, "n": n, "link": rng.choice([3.8950534e-5, 5e-4, 2e-3])}
    if kind == "direct":
        return {"kind": kind, "n": _log_int(rng, 16384, 1048576),
                "targets": _log_int(rng, 512, 16384), "phi": rng.random() < 0.5}
    return {"kind": kind, "n": _log_int(rng, 4096, 1048576)}


# ----------------------------------------------------------------- inputs
def _disk(n, seed, r_min, r_max, sigma_e=0.01, sigma_i=0.005):
    """Keplerian disk in the XZ plane: x, v as (3, n) float64 CUDA tensors."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 2654435761 % (1 << 62) + n)
    u = torch.rand((6, n), dtype=torch.float64, device="cuda", generator=g)
    a = (math.sqrt(r_min) + u[0] * (math.sqrt(r_max) - math.sqrt(r_min))) ** 2
    e = (sigma_e * torch.sqrt(-2.0 * torch.log1p(-u[1]))).clamp(max=0.3)
    inc = (sigma_i * torch.sqrt(-2.0 * torch.log1p(-u[2]))).clamp(max=0.3)
    om, w, big_m = (2.0 * math.pi * u[k] for k in (3, 4, 5))
    ec = big_m.clone()
    for _ in range(6):  # Kepler's equation
        ec = ec - (ec - e * torch.sin(ec) - big_m) / (1.0 - e * torch.cos(ec))
    ce, se, q = torch.cos(ec), torch.sin(ec), torch.sqrt(1.0 - e * e)
    p, s = a * (ce - e), a * q * se
    f = torch.sqrt(1.0 / a) / (1.0 - e * ce)
    dp, ds = -f * se, f * q * ce
    cw, sw, co, so = torch.cos(w), torch.sin(w), torch.cos(om), torch.sin(om)
    ci, si = torch.cos(inc), torch.sin(inc)
    px, pz, py = co * cw - so * sw * ci, so * cw + co * sw * ci, sw * si
    qx, qz, qy = -co * sw - so * cw * ci, -so * sw + co * cw * ci, cw * si
    x = torch.stack([p * px + s * qx, p * py + s * qy, p * pz + s * qz])
    v = torch.stack([dp * px + ds * qx, dp * py + ds * qy, dp * pz + ds * qz])
    return x, v


def _ensemble_disks(c):
    rng = np.random.default_rng(c["layout"])
    lo, hi = math.log(c["n_lo"]), math.log(c["n_hi"])
    return [{"n": int(round(math.exp(rng.uniform(lo, hi)))), "perturber_enabled": 1,
             "perturber_mass_mjup": float(np.float32(math.exp(rng.uniform(math.log(0.3),
                                                                          math.log(10.0))))),
             "perturber_radius_au": float(np.float32(rng.uniform(5.0, 30.0))),
             "perturber_phase0": float(np.float32(rng.uniform(0.0, 2.0 * math.pi)))}
            for _ in range(c["disks"])]


def _physics(c):
    """The step's physical parameters, in one form for every kind."""
    k = c["kind"]
    p = {"mass": 1e-8, "eps": 1e-3, "theta": 0.5, "dt": 0.005, "r_coll": 0.0, "drag": 0.0,
         "pert_mass": 0.0, "pert_radius": 5.2, "phase0": 0.0, "r_min": 0.5, "r_max": 5.0}
    if k == "gradient":
        p.update(drag=1e-3, pert_mass=3.0, pert_radius=10.0, phase0=0.5)
    if k in ("host", "direct"):
        p.update(mass=1e-9, eps=5e-4, dt=0.002, r_min=0.3, r_max=30.0)
    p.update({q: c[q] for q in p if q in c})
    return p


def _params(p, **kw):
    return nb.sim_params(dt=p["dt"], theta=p["theta"], softening=p["eps"], star_mass=1.0,
                         r_coll=p["r_coll"], restitution=0.0, gas_drag_rate=p["drag"],
                         perturber_enabled=int(p["pert_mass"] > 0.0),
                         perturber_mass_mjup=p["pert_mass"],
                         perturber_radius_au=p["pert_radius"], perturber_phase0=p["phase0"], **kw)


def _inputs(c, seed):
    """(x, v) of the case's bodies in the type its entry point takes."""
    p = _physics(c)
    n = sum(d["n"] for d in _ensemble_disks(c)) if c["kind"] == "ensemble" else c["n"]
    x, v = _disk(n, seed, p["r_min"], p["r_max"])
    if c["kind"] in ("phases", "fof", "host") or c.get("state") == "f32":
        x, v = x.float(), v.float()
    return x, v


def prepare(case, seed):
    c, k, p = case, case["kind"], _physics(case)
    x, v = _inputs(c, seed)
    n = x.shape[1]
    mass = torch.full((n,), p["mass"], dtype=torch.float32, device="cuda")
    s = {"case": c, "n": n, "p": p}
    if k == "step":
        s["sim"] = nb.Sim(_params(p, state_precision=STATES[c["state"]]), n)
        s["sim"].set_state(*x, *v, mass)
        s["out"] = {q: torch.empty(n, dtype=x.dtype, device="cuda") for q in KEYS}
        if c["state"] == "f32":
            s["out"].update({q: torch.empty(n, device="cuda") for q in ACC})
    elif k == "ensemble":
        s["sim"] = nb.Ensemble(_params(p, state_precision=nb.STATE_F64), _ensemble_disks(c))
        s["sim"].set_state(*x, *v, mass)
        s["out"] = {q: torch.empty(n, dtype=torch.float64, device="cuda") for q in KEYS}
        s["out"].update({q: torch.empty(n, device="cuda") for q in ACC})
    elif k == "gradient":
        s["engine"] = nb.Adjoint(_params(p), n, c["steps"], c["mode"], c["every"] or 50)
        s.update(x=x, v=v, mass=mass)
    elif k == "phases":
        s["pd"] = nb.allocate_particles_gpu(n)
        for q, t in zip(KEYS, (*x, *v)):
            s["pd"].arrays[q].copy_(t)
        s["pd"].arrays["mass"].copy_(mass)
        s["tree"] = nb.Octree(n)
        cfg = nb.default_config()
        cfg.perturber_enabled = int(p["pert_mass"] > 0.0)
        cfg.perturber_mass_mjup, cfg.perturber_radius_AU = p["pert_mass"], p["pert_radius"]
        cfg.perturber_phase0, cfg.star_mass_msun = p["phase0"], 1.0
        s["pert"], s["step"] = nb.make_perturber(cfg), 0
        s["tree"].reset()
        s["tree"].bbox(s["pd"])
        s["tree"].build(s["pd"])
        s["tree"].summarize()
        s["tree"].force(s["pd"], p["theta"], p["eps"], 1.0)
        if s["pert"].enabled:
            q = s["pert"]
            nb.perturber_force(s["pd"], q.x, q.y, q.z, q.mass_msun, p["eps"])
    elif k == "fof":
        s["tree"], s["x"] = nb.Octree(n), x
    elif k == "direct":
        s.update(x=x, mass=mass, targets=_targets(c, seed))
    elif k == "host":
        sim = nb.Sim(_params(p), n)
        sim.set_state(*x, *v, mass)
        got = sim.get_state()
        host = {q: torch.empty(n, pin_memory=True) for q in KEYS + ACC}
        for q in KEYS + ACC:
            host[q].copy_(torch.from_numpy(got[q]))
        s["sim"], s["pin"] = sim, (host, mass.cpu().pin_memory())
        s["host"] = {q: t.numpy() for q, t in host.items()}
        s["mass"] = s["pin"][1].numpy()
    return s


def _targets(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 77)
    return torch.randperm(c["n"], device="cuda", generator=g)[:min(c["targets"], c["n"])].int()


# ------------------------------------------------------------------- runs
def _check(rc):
    if rc != nb.NBODY_OK:
        raise nb.NBodyError(rc, nb.lib.nbody_last_error().decode())


def run(state):
    s, c, p = state, state["case"], state["p"]
    k = c["kind"]
    if k == "step":
        s["sim"].step(c["steps"])
        ptr = {q: t.data_ptr() for q, t in s["out"].items()}
        pos = [ptr[q] for q in KEYS]
        if c["state"] == "f32":  # the read-out into device memory, through the C interface
            _check(nb.lib.nbody_sim_get_state(s["sim"].h, *pos, *[ptr[q] for q in ACC], 1))
        else:
            _check(nb.lib.nbody_sim_get_state_f64(s["sim"].h, *pos, 1))
        return s["out"]
    if k == "ensemble":
        s["sim"].step(c["steps"])
        _check(nb.lib.nbody_ensemble_get_state_f64(
            s["sim"].h, *[s["out"][q].data_ptr() for q in KEYS + ACC], 1))
        return s["out"]
    if k == "gradient":
        x0, v0 = s["x"].requires_grad_(), s["v"].requires_grad_()
        pm = torch.tensor(p["pert_mass"], dtype=torch.float64, requires_grad=True)
        pr = torch.tensor(p["pert_radius"], dtype=torch.float64, requires_grad=True)
        x, v = nb.disk_trajectory(s["engine"], x0, v0, pm, pr, s["mass"])
        loss = nb.eccentricity_loss(x, v, s["mass"], 1.0, 2.0)
        gx, gv, gm, gr = torch.autograd.grad(loss, (x0, v0, pm, pr))
        return {"x": x.detach(), "v": v.detach(), "loss": loss.detach(), "gx": gx, "gv": gv,
                "gm": gm, "gr": gr}
    if k == "phases":
        pd, tree, q = s["pd"], s["tree"], s["pert"]
        s["step"] += 1
        nb.half_kick(pd, 0.5 * p["dt"])
        nb.drift(pd, p["dt"])
        nb.reset_acceleration(pd)
        tree.reset()
        tree.bbox(pd)
        tree.build(pd)
        tree.summarize()
        tree.sort()
        tree.force(pd, p["theta"], p["eps"], 1.0)
        if q.enabled:
            nb.update_perturber(q, s["step"] * p["dt"])
            nb.perturber_force(pd, q.x, q.y, q.z, q.mass_msun, p["eps"])
        if p["r_coll"] > 0.0:
            tree.collide(pd, p["r_coll"], 0.0)
        nb.half_kick(pd, 0.5 * p["dt"])
        nb.gas_drag(pd, p["drag"], p["dt"], 1.0)
        return {f: pd.arrays[f] for f in KEYS + ACC}
    if k == "fof":
        labels, agg, groups = s["tree"].fof(*s["x"], c["link"])
        return {"labels": labels, "agg_size": agg, "groups": groups}
    if k == "direct":
        ax, ay, az, phi = nb.direct_f64(*s["x"], s["mass"], p["eps"], s["targets"],
                                        want_phi=c["phi"])
        return {"ax": ax, "ay": ay, "az": az, **({"phi": phi} if c["phi"] else {})}
    s["sim"].step_host(s["host"], s["mass"], 1)
    return s["host"]


# ------------------------------------------------------------------- work
def _tree_flops(n):
    """A monopole walk at theta = 0.5 meets about 20 log2(n) sources a body, 19 FLOP each."""
    return 19.0 * 20.0 * math.log2(max(n, 2)) * n


def work(case):
    c, k = case, case["kind"]
    if k == "step":
        b = {"f32": 4, "f64": 8, "f32x2": 8}[c["state"]]
        out = 24 if c["state"] == "f32" else 48
        return {"bytes": c["n"] * (6.0 * b + 4 + out + (12 if b == 4 else 0)),
                "flops": c["steps"] * _tree_flops(c["n"])}
    if k == "ensemble":
        sizes = [d["n"] for d in _ensemble_disks(c)]
        return {"bytes": sum(sizes) * (48.0 + 4 + 48 + 12),
                "flops": c["steps"] * sum(_tree_flops(n) for n in sizes)}
    if k == "gradient":  # forward, and a product with the Jacobian of twice its work
        return {"bytes": c["n"] * (48.0 + 4 + 48 + 48),
                "flops": 3.0 * c["steps"] * _tree_flops(c["n"])}
    if k == "phases":
        return {"bytes": c["n"] * (40.0 + 36), "flops": _tree_flops(c["n"])}
    if k == "fof":
        return {"bytes": c["n"] * (12.0 + 6), "flops": 8.0 * c["n"] * math.log2(c["n"])}
    if k == "direct":
        t = min(c["targets"], c["n"])
        return {"bytes": c["n"] * 28.0 + t * (4 + (32.0 if c["phi"] else 24.0)),
                "flops": 20.0 * t * c["n"]}
    return {"bytes": c["n"] * (40.0 + 36), "flops": _tree_flops(c["n"])}


# ------------------------------------------------------------------ exact
def _rows(nt, n):
    step = max(1, (1 << 25) // n)
    return [(a, min(nt, a + step)) for a in range(0, nt, step)]


def _gravity(x, m, eps, v=None, r_coll=0.0, targets=None, phi=False):
    """Direct-sum self-gravity on the targets (every body by default); with
    r_coll also the collision impulses of the approaching pairs (restitution 0)."""
    n = x.shape[1]
    idx = torch.arange(n, device=x.device) if targets is None else targets.long()
    acc = torch.zeros((3, idx.numel()), dtype=x.dtype, device=x.device)
    pot = torch.zeros(idx.numel(), dtype=x.dtype, device=x.device)
    dv = torch.zeros_like(acc)
    xt = x.t().contiguous()
    for a, b in _rows(idx.numel(), n):
        me = idx[a:b]
        r2 = torch.zeros((b - a, n), dtype=x.dtype, device=x.device)
        for k in range(3):
            d = x[k][None, :] - x[k][me][:, None]
            r2.addcmul_(d, d)
        if r_coll > 0.0:
            close = torch.nonzero(r2 < r_coll * r_coll)
            close = close[me[close[:, 0]] != close[:, 1]]
            if close.numel():
                i, j = me[close[:, 0]], close[:, 1]
                d = x[:, j] - x[:, i]
                d = d / (torch.sqrt((d * d).sum(0)) + 1e-10)
                dvn = ((v[:, j] - v[:, i]) * d).sum(0).clamp(max=0.0)
                dv.index_add_(1, i, 0.5 * dvn * d)
        inv = r2.add_(eps * eps).rsqrt_()
        inv[torch.arange(b - a, device=x.device), me] = 0.0
        if phi:
            pot[a:b] = -(inv @ m)
        f = (inv * inv).mul_(inv).mul_(m[None, :])
        acc[:, a:b] = (f @ xt).t() - x[:, me] * f.sum(1)
    return acc, dv, pot


def _central(x, eps, pert):
    """Star and (x, y, z, mass) perturber pulls."""
    a = -x / ((x * x).sum(0) + eps * eps) ** 1.5
    if pert is not None:
        d = torch.stack([pert[0] - x[0], pert[1] - x[1], pert[2] - x[2]])
        a = a + pert[3] * d / ((d * d).sum(0) + eps * eps) ** 1.5
    return a


def _drag(x, v, decay):
    r = torch.sqrt(x[0] ** 2 + x[2] ** 2)
    ux, uz = x[0] / r, x[2] / r
    vr, vp = v[0] * ux + v[2] * uz, -v[0] * uz + v[2] * ux
    kep = torch.where(vp >= 0, 1.0, -1.0) / torch.sqrt(r)
    vr, vp = vr * decay, kep + (vp - kep) * decay
    return torch.stack([vr * ux - vp * uz, v[1] * decay, vr * uz + vp * ux])


def _f(v):
    return float(np.float32(v))


def _perturber(p, mass, radius, t):
    if not p["pert_mass"] > 0.0:
        return None
    if not torch.is_tensor(radius):
        mass, radius = torch.tensor(mass, dtype=torch.float64), torch.tensor(radius, dtype=torch.float64)
    phi = _f(p["phase0"]) + t / radius ** 1.5
    return radius * torch.cos(phi), 0.0 * radius, radius * torch.sin(phi), MJUP * mass


def _steps(p, x, v, m, steps, gravity, mass, radius):
    """`steps` KDK steps in FP64; gravity(x, v) -> (acceleration, impulse)."""
    dt, eps, decay = _f(p["dt"]), _f(p["eps"]), math.exp(-_f(p["drag"]) * _f(p["dt"]))
    acc = gravity(x, None)[0] + _central(x, eps, _perturber(p, mass, radius, 0.0))
    for k in range(steps):
        v = v + 0.5 * dt * acc
        x = x + dt * v
        g, dv = gravity(x, v)
        acc = g + _central(x, eps, _perturber(p, mass, radius, (k + 1) * dt))
        v = v + dv + 0.5 * dt * acc
        if p["drag"] > 0.0:
            v = _drag(x, v, decay)
    return x, v, acc


class _DirectGravity(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, m, eps):
        ctx.save_for_backward(x, m)
        ctx.eps = eps
        return _gravity(x, m, eps)[0]

    @staticmethod
    def backward(ctx, lam):
        (x, m), n = ctx.saved_tensors, lam.shape[1]
        g = torch.zeros_like(x)
        for a, b in _rows(n, n):
            d = [x[k][None, :] - x[k][a:b][:, None] for k in range(3)]
            w = [m[a:b][:, None] * lam[k][None, :] - m[None, :] * lam[k][a:b][:, None]
                 for k in range(3)]
            i2 = (d[0] * d[0]).addcmul_(d[1], d[1]).addcmul_(d[2], d[2]).add_(ctx.eps ** 2).reciprocal_()
            i3 = i2 * i2.sqrt()
            dw = (d[0] * w[0]).addcmul_(d[1], w[1]).addcmul_(d[2], w[2]).mul_(i2).mul_(3.0)
            for k in range(3):
                g[k, a:b] = ((w[k] - d[k] * dw) * i3).sum(1)
        return g, None, None


def _seconds(pairs, passes):
    return passes * pairs * 220.0 / 6e12


def exact(case, seed):
    c, k, p = case, case["kind"], _physics(case)
    if k == "fof" or k == "host" and _seconds(c["n"] ** 2, 2) > 15.0:
        return None
    if k in ("step", "phases") and _seconds(c["n"] ** 2, c.get("steps", 1) + 1) > 15.0:
        return None
    if k == "gradient" and _seconds(c["n"] ** 2, 5 * c["steps"]) > 15.0:
        return None
    if k == "ensemble" and _seconds(sum(d["n"] ** 2 for d in _ensemble_disks(c)),
                                    c["steps"] + 1) > 15.0:
        return None
    x, v = (t.double() for t in _inputs(c, seed))
    m = torch.full((x.shape[1],), _f(p["mass"]), dtype=torch.float64, device="cuda")
    eps, rc = _f(p["eps"]), _f(p["r_coll"])
    if k == "direct":  # this entry point takes its softening as a double
        acc, _, phi = _gravity(x, m, p["eps"], targets=_targets(c, seed), phi=c["phi"])
        return {"ax": acc[0], "ay": acc[1], "az": acc[2], **({"phi": phi} if c["phi"] else {})}
    if k == "gradient":
        x, v = x.requires_grad_(), v.requires_grad_()
        pm = torch.tensor(p["pert_mass"], dtype=torch.float64, requires_grad=True)
        pr = torch.tensor(p["pert_radius"], dtype=torch.float64, requires_grad=True)
        x1, v1, _ = _steps(p, x, v, m, c["steps"],
                           lambda x, v: (_DirectGravity.apply(x, m, eps), 0.0), pm, pr)
        r = torch.sqrt((x1 * x1).sum(0))
        e = ((v1 * v1).sum(0) - 1.0 / r) * x1 - (x1 * v1).sum(0) * v1
        w = m * (r < 2.0)
        loss = (w * (e * e).sum(0)).sum() / w.sum()
        gx, gv, gm, gr = torch.autograd.grad(loss, (x, v, pm, pr))
        return {"x": x1.detach(), "v": v1.detach(), "loss": loss.detach(), "gx": gx, "gv": gv,
                "gm": gm, "gr": gr}

    def one(x, v, m, mass, radius, phase0):
        q = dict(p, phase0=phase0, pert_mass=mass)
        return _steps(q, x, v, m, c.get("steps", 1),
                      lambda x, v: _gravity(x, m, eps, v, rc if v is not None else 0.0)[:2],
                      mass, radius)

    if k == "ensemble":
        parts, at = [], 0
        for d in _ensemble_disks(c):
            sl = slice(at, at + d["n"])
            parts.append(one(x[:, sl], v[:, sl], m[sl], d["perturber_mass_mjup"],
                             d["perturber_radius_au"], d["perturber_phase0"]))
            at += d["n"]
        x, v, acc = (torch.cat([q[i] for q in parts], 1) for i in range(3))
    else:
        x, v, acc = one(x, v, m, _f(p["pert_mass"]), _f(p["pert_radius"]), p["phase0"])
    out = dict(zip(KEYS, (*x, *v)))
    if k != "step" or c["state"] == "f32":
        out.update(zip(ACC, acc))
    return out
