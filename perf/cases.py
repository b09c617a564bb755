"""What a user of the engine has it do, as cases of measured size.

Four kinds of call, all through the Python face of the public interface:

  steps     a run between two outputs: kick-drift-kick steps through the Backend calls, then the
            diagnostics (where the case logs them) and the download of the bodies for a snapshot
  forces    one force evaluation of a new snapshot: upload, forces with the potential, read back
  adjoint   one step of a fit: upload the current initial conditions, forward pass, backward pass
  ensemble  a batch of independent clusters advanced together in one call, then the download

Sizes follow the repository's workloads (Plummer 16384 and 65536 bodies direct, the 1e6-body disk,
the collision of two disks, clusters of 1024 to 131072 bodies) and fill the range between and below
them with odd sizes. Initial conditions have the distributions of the package's scenarios, drawn on
the GPU so that making them is quick.
"""
import math

import numpy as np
import torch

import lettuce_simulate_physics_gb300 as L
from lettuce_simulate_physics_gb300.ensemble import Ensemble

FIELDS = ("x", "y", "z", "vx", "vy", "vz", "m")


def listed():
    return [
        # A star cluster small enough that every call is latency: logs its energy, then a snapshot.
        dict(name="direct_1k", kind="steps", method="direct", scene="plummer", n=1000, eps=0.01, theta=0.0, dt=1e-3,
             steps=20, log="end"),
        # An odd size, with the potential in every force call (a run that logs its energy each step).
        dict(name="direct_5k_energy", kind="steps", method="direct", scene="cube", n=5001, eps=0.02, theta=0.0,
             dt=1e-3, steps=10, log="every"),
        # The direct workload: a Plummer sphere of 16384 bodies, ten steps.
        dict(name="direct_16k", kind="steps", method="direct", scene="plummer", n=16384, eps=0.01, theta=0.0, dt=1e-3,
             steps=10, log="no"),
        # The largest direct runs, one body past a tile boundary.
        dict(name="direct_65k", kind="steps", method="direct", scene="plummer", n=65537, eps=0.01, theta=0.0, dt=1e-3,
             steps=2, log="no"),
        # The smallest trees in use (just above where direct summation is still the better choice).
        dict(name="tree_8k", kind="steps", method="tree", scene="plummer", n=8191, eps=0.01, theta=0.6, dt=1e-3,
             steps=10, log="no"),
        # An ordinary cluster run with its energy in the log, at the ensembles' opening angle.
        dict(name="tree_100k", kind="steps", method="tree", scene="plummer", n=100003, eps=0.01, theta=0.5, dt=1e-3,
             steps=4, log="end"),
        # The headline workload: the 1e6-body exponential disk.
        dict(name="tree_1m_disk", kind="steps", method="tree", scene="disk", n=1000000, eps=0.005, theta=0.6, dt=5e-4,
             steps=2, log="no"),
        # The largest run: the collision of two 8e6-body disks.
        dict(name="tree_16m_collision", kind="steps", method="tree", scene="collision", n=16000000, eps=0.005,
             theta=0.6, dt=5e-4, steps=1, log="no"),
        # A snapshot analysed once: everything on new inputs, the tree's first build among it.
        dict(name="forces_131k", kind="forces", method="tree", scene="disk", n=131071, eps=0.005, theta=0.6),
        # Fitting initial conditions of the 65536-body Plummer sphere: forward and backward.
        dict(name="adjoint_65k", kind="adjoint", method="direct", scene="plummer", n=65536, eps=0.01, theta=0.0,
             dt=1e-3, steps=8, every=4),
        # The same through tree forces: a small collision, frozen interaction lists.
        dict(name="adjoint_tree_200k", kind="adjoint", method="tree", scene="collision", n=200000, eps=0.005,
             theta=0.6, dt=5e-4, steps=4, every=2),
        # A parameter scan: clusters of 1024 to 131072 bodies, direct and tree systems side by side.
        dict(name="ensemble_96", kind="ensemble", systems=96, lo=1024, hi=131072, theta=0.5, dt=1e-3, steps=8),
    ]


def _between(rng, lo, hi):
    """Log-uniform whole number."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "forces", "adjoint", "ensemble"])
    if kind == "ensemble":
        hi = _between(rng, 4096, 131072)
        return dict(kind=kind, systems=_between(rng, 12, 96), lo=1024, hi=hi, theta=rng.choice([0.4, 0.5, 0.6]),
                    dt=1e-3, steps=rng.randint(3, 8))
    if kind == "adjoint":
        if rng.random() < 0.6:
            steps = rng.randint(2, 8)
            return dict(kind=kind, method="direct", scene="plummer", n=_between(rng, 1024, 65536), eps=0.01,
                        theta=0.0, dt=1e-3, steps=steps, every=rng.randint(1, steps))
        steps = rng.randint(2, 4)
        return dict(kind=kind, method="tree", scene=rng.choice(["plummer", "disk", "collision"]),
                    n=_between(rng, 10000, 200000), eps=0.01, theta=0.6, dt=5e-4, steps=steps,
                    every=rng.randint(1, steps))
    tree = kind == "forces" or rng.random() < 0.6
    if kind == "forces":
        n = _between(rng, 10000, 1000000)
        return dict(kind=kind, method="tree", scene=rng.choice(["plummer", "disk", "collision"]), n=n, eps=0.01,
                    theta=rng.choice([0.5, 0.6, 0.7]))
    if tree:
        n = _between(rng, 5000, 8000000)
        return dict(kind=kind, method="tree", scene=rng.choice(["plummer", "disk", "collision"]), n=n, eps=0.01,
                    theta=rng.choice([0.5, 0.6, 0.7]), dt=5e-4, steps=1 if n > 2000000 else rng.randint(1, 8),
                    log=rng.choice(["no", "no", "end"]))
    n = _between(rng, 500, 65537)
    return dict(kind=kind, method="direct", scene=rng.choice(["plummer", "cube"]), n=n, eps=0.01, theta=0.0, dt=1e-3,
                steps=rng.randint(1, 3) if n > 20000 else rng.randint(4, 20), log=rng.choice(["no", "end", "every"]))


# ---- inputs -----------------------------------------------------------------------------------
def _interp(u, grid, cdf):
    """x with cdf(x) = u, linear between grid points."""
    k = torch.searchsorted(cdf, u).clamp(1, len(cdf) - 1)
    c0, c1 = cdf[k - 1], cdf[k]
    t = torch.where(c1 > c0, (u - c0) / (c1 - c0), torch.zeros_like(u))
    return grid[k - 1] + t * (grid[k] - grid[k - 1])


def _directions(g, n):
    z = 2 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 1
    phi = 2 * math.pi * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    s = torch.sqrt((1 - z * z).clamp_min(0))
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z])


def _plummer(n, g):
    """Equal masses 1/n in Henon units, truncated at ten scale lengths."""
    a, cut = 3 * math.pi / 16, 10.0
    top = (1 + 1 / cut ** 2) ** -1.5
    u = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * top).clamp_min(1e-12)
    r = a / torch.sqrt(u ** (-2 / 3) - 1)
    q = torch.linspace(0, 1, 8193, device="cuda", dtype=torch.float64)
    cdf = torch.cumsum(q * q * (1 - q * q) ** 3.5, 0)
    q = _interp(torch.rand(n, generator=g, device="cuda", dtype=torch.float64), q, cdf / cdf[-1])
    v = q * math.sqrt(2 / a) * (1 + (r / a) ** 2) ** -0.25
    return r * _directions(g, n), v * _directions(g, n), torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)


def _cube(n, g):
    x = 2 * torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64) - 1
    v = 2 * torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64) - 1
    return x, v, (0.5 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64)) / n


def _disk(n, g):
    """Exponential disk (scale length 1, cut at 10, sech^2 of height 0.1) around a core of mass 1."""
    ns = n - 1
    x = torch.linspace(0, 10, (1 << 16) + 1, device="cuda", dtype=torch.float64)
    cdf = 1 - (1 + x) * torch.exp(-x)
    R = _interp(torch.rand(ns, generator=g, device="cuda", dtype=torch.float64) * cdf[-1], x, cdf)
    R = torch.sort(R).values.clamp_min(1e-12)
    phi = 2 * math.pi * torch.rand(ns, generator=g, device="cuda", dtype=torch.float64)
    z = 0.1 * torch.atanh((2 * torch.rand(ns, generator=g, device="cuda", dtype=torch.float64) - 1).clamp(-1 + 1e-14, 1 - 1e-14))
    vc = torch.sqrt((1 + torch.arange(1, n, device="cuda", dtype=torch.float64) / ns) / R)
    c, s = torch.cos(phi), torch.sin(phi)
    noise = 0.05 * vc * torch.randn((3, ns), generator=g, device="cuda", dtype=torch.float64)
    pos = torch.zeros((3, n), device="cuda", dtype=torch.float64)
    vel = torch.zeros((3, n), device="cuda", dtype=torch.float64)
    pos[:, 1:] = torch.stack([R * c, R * s, z])
    vel[:, 1:] = torch.stack([-vc * s, vc * c, torch.zeros_like(vc)]) + noise
    m = torch.full((n,), 1.0 / ns, device="cuda", dtype=torch.float64)
    m[0] = 1.0
    return pos, vel, m


def _collision(n, g):
    """Two disks inclined by 45 and 30 degrees, 20 apart on a parabolic approach (pericentre 3)."""
    sizes = (n // 2, n - n // 2)
    r0, vt = 20.0, math.sqrt(2 * 4 * 3.0) / 20
    vr = -math.sqrt(2 * 4 / r0 - vt * vt)
    parts = []
    for k, (ns, incl) in enumerate(zip(sizes, (45.0, 30.0))):
        pos, vel, m = _centred(*_disk(ns, g))
        c, s = math.cos(math.radians(incl)), math.sin(math.radians(incl))
        side = 0.5 if k == 0 else -0.5
        out = []
        for w, shift in ((pos, (r0, 0.0, 0.0)), (vel, (vr, vt, 0.0))):
            w = torch.stack([w[0], w[1] * c - w[2] * s, w[1] * s + w[2] * c])
            out.append(w + side * torch.tensor(shift, device="cuda", dtype=torch.float64)[:, None])
        parts.append((*out, m))
    return tuple(torch.cat([p[q] for p in parts], dim=-1) for q in range(3))


def _centred(pos, vel, m):
    M = m.sum()
    return pos - (pos * m).sum(1, keepdim=True) / M, vel - (vel * m).sum(1, keepdim=True) / M, m


def _bodies(scene, n, g):
    make = {"plummer": _plummer, "cube": _cube, "disk": _disk, "collision": _collision}[scene]
    cols = make(n, g)
    pos, vel, m = (t.float().cpu().numpy() for t in (cols if scene == "cube" else _centred(*cols)))
    return L.Bodies(*pos, *vel, m, np.arange(n, dtype=np.uint32))


def _pinned(n):
    """Bodies in page-locked host memory, for the downloads."""
    buf = torch.empty((8, n), dtype=torch.float32, pin_memory=True).numpy()
    return L.Bodies(*buf[:7], buf[7].view(np.uint32))


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _params(case):
    return L.ForceParams(G=1.0, eps=case["eps"], theta=case["theta"],
                         method=L.ForceMethod.tree if case["method"] == "tree" else L.ForceMethod.direct)


def _ensemble_inputs(case, seed):
    g = _generator(seed)
    # The scan's plan of sizes, log-uniform and the same for every seed.
    u = ((np.arange(case["systems"]) + 0.5) * (math.sqrt(5.0) - 1) / 2) % 1.0
    counts = np.floor(case["lo"] * (case["hi"] / case["lo"]) ** u).astype(np.int64)
    parts = [_centred(*_plummer(int(c), g)) for c in counts]
    pos, vel, m = (torch.cat([p[q] for p in parts], dim=-1).float().cpu().numpy() for q in range(3))
    b = L.Bodies(*pos, *vel, m, np.arange(int(counts.sum()), dtype=np.uint32))
    eps = 0.01 * (counts / 16384.0) ** (-1.0 / 3.0)
    return b, counts, eps, np.where(counts <= 8192, 0, 1)


def prepare(case, seed):
    if case["kind"] == "ensemble":
        b, counts, eps, method = _ensemble_inputs(case, seed)
        en = Ensemble(0)
        en.upload(b, counts, eps, np.full(len(counts), case["theta"]), method)
        # A scan advances its batch call after call: the first call's forces and sizes are there.
        en.run(case["dt"], case["steps"], use_graph=True)
        return dict(case=case, en=en)
    b = _bodies(case["scene"], case["n"], _generator(seed))
    be = L.CudaBackend(0)
    state = dict(case=case, be=be, p=_params(case), bodies=b)
    if case["kind"] == "steps":
        be.upload(b)
        be.compute_forces(state["p"], case["log"] == "every")
        state["out"] = _pinned(case["n"])
        del state["bodies"]
    elif case["kind"] == "forces":
        state["out"] = _pinned(case["n"])
    else:
        # The target: where the bodies would be after free flight, shifted a little.
        t = case["dt"] * case["steps"]
        state["target"] = b.pos64() + t * b.vel64() + 1e-3
    return state


# ---- one pass ---------------------------------------------------------------------------------
def _outputs(b):
    return {f: getattr(b, f) for f in FIELDS} | {"id": b.id.view(np.int32)}


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        state["en"].run(case["dt"], case["steps"], use_graph=True)
        b = state["en"].download()
        return _outputs(b)
    be, p = state["be"], state["p"]
    if case["kind"] == "adjoint":
        be.upload(state["bodies"])
        be.adjoint_forward(p, case["dt"], case["steps"], case["every"])
        loss, gx, gv, gm = be.adjoint_backward(state["target"])
        # The parameters are float32 columns: so are the gradients that an optimiser takes.
        return {"loss": loss, "gx": gx.astype(np.float32), "gv": gv.astype(np.float32), "gm": gm.astype(np.float32)}
    if case["kind"] == "forces":
        be.upload(state["bodies"])
        be.compute_forces(p, True)
        a = be.accel()
        b = be.download(state["out"])  # the ids that go with them
        return {"a": a[:3], "phi": a[3], "id": b.id.view(np.int32)}
    for k in range(case["steps"]):
        be.kick(0.5 * case["dt"])
        be.drift(case["dt"])
        be.compute_forces(p, case["log"] == "every" or (case["log"] == "end" and k == case["steps"] - 1))
        be.kick(0.5 * case["dt"])
    out = {}
    if case["log"] != "no":
        d = be.diagnostics()
        out = {"ke": d.ke, "pe": d.pe}
    b = be.download(state["out"])
    return out | _outputs(b)


# ---- the same in 64 bits ----------------------------------------------------------------------
def _accel(x, m, eps, phi=False):
    """(3, n) accelerations, and the potential, of all bodies by direct summation in FP64."""
    n = x.shape[1]
    a = torch.empty_like(x)
    pot = torch.empty_like(m)
    rows = max(1, min(n, (1 << 25) // n))
    xm = torch.cat([x * m, m[None]]).T.contiguous()
    for i in range(0, n, rows):
        xi = x[:, i:i + rows]
        r2 = torch.full((xi.shape[1], n), eps * eps, device="cuda", dtype=torch.float64)
        for c in range(3):
            d = x[c][None, :] - xi[c][:, None]
            r2.addcmul_(d, d)
        inv = torch.rsqrt(r2)
        if phi:
            pot[i:i + rows] = m[i:i + rows] / eps - inv @ m
        s = inv.mul(inv).mul_(inv) @ xm
        a[:, i:i + rows] = s[:, :3].T - xi * s[:, 3]
    return a, pot


def _vjp(x, m, w, eps):
    """Gradient of sum_k w_k . a_k with respect to positions and masses, FP64."""
    n = x.shape[1]
    gx = torch.empty_like(x)
    gm = torch.empty_like(m)
    rows = max(1, min(n, (1 << 25) // n))
    for i in range(0, n, rows):
        xi, wi, mi = x[:, i:i + rows], w[:, i:i + rows], m[i:i + rows]
        d = [x[c][None, :] - xi[c][:, None] for c in range(3)]
        r2 = torch.full((xi.shape[1], n), eps * eps, device="cuda", dtype=torch.float64)
        for c in range(3):
            r2.addcmul_(d[c], d[c])
        inv = torch.rsqrt(r2)
        inv3 = inv * inv * inv
        dwj = sum(d[c] * w[c][None, :] for c in range(3))
        dwi = sum(d[c] * wi[c][:, None] for c in range(3))
        gm[i:i + rows] = -(dwj * inv3).sum(1)
        # M(d) u = u / s^3 - 3 d (d . u) / s^5 with u = m_i w_j - m_j w_i
        du = (mi[:, None] * dwj - m[None, :] * dwi).mul_(inv3).mul_(inv).mul_(inv)
        s3m = inv3 @ m
        for c in range(3):
            gx[c, i:i + rows] = mi * (inv3 @ w[c]) - wi[c] * s3m - 3 * (du * d[c]).sum(1)
    return gx, gm


def _morton_order(x):
    """The order of the bodies by their 63-bit Morton keys."""
    lo = x.min(1, keepdim=True).values
    side = float((x.max(1, keepdim=True).values - lo).max()) * (1 + 1e-6)
    q = ((x - lo) * ((1 << 21) / side)).to(torch.int64).clamp(0, (1 << 21) - 1)
    key = torch.zeros(x.shape[1], dtype=torch.int64, device="cuda")
    for bit in range(21):
        for c in range(3):
            key |= ((q[c] >> bit) & 1) << (3 * bit + 2 - c)
    return torch.argsort(key, stable=True)


def _state64(b):
    t = lambda *f: torch.tensor(np.stack([getattr(b, k) for k in f]).astype(np.float64), device="cuda")  # noqa: E731
    return t("x", "y", "z"), t("vx", "vy", "vz"), t("m")[0]


def _columns(x, v, m):
    return {f: c.cpu().numpy() for f, c in zip(FIELDS, (*x, *v, m))} | {"id": None}


def exact(case, seed):
    if case["kind"] == "ensemble":
        b, counts, eps, method = _ensemble_inputs(case, seed)
        if method.any() or float((counts.astype(np.float64) ** 2).sum()) * case["steps"] > 2e10:
            return None  # tree systems come back in an order of their own
        x, v, m = _state64(b)
        off = 0
        for c, e in zip(counts, eps):
            s = slice(off, off + int(c))
            xs, vs, ms = x[:, s].clone(), v[:, s].clone(), m[s]
            a, _ = _accel(xs, ms, float(e))
            for _ in range(2 * case["steps"]):  # prepare's run and the pass
                vs += 0.5 * case["dt"] * a
                xs += case["dt"] * vs
                a, _ = _accel(xs, ms, float(e))
                vs += 0.5 * case["dt"] * a
            x[:, s], v[:, s] = xs, vs
            off += int(c)
        return _columns(x, v, m)
    n, eps = case["n"], case["eps"]
    pairs = float(n) * n
    if case["kind"] == "forces":
        if pairs > 3e10:
            return None
        x, v, m = _state64(_bodies(case["scene"], n, _generator(seed)))
        o = _morton_order(x)
        x, m = x[:, o], m[o]
        a, phi = _accel(x, m, eps, phi=True)
        return {"a": a.cpu().numpy(), "phi": phi.cpu().numpy(), "id": None}
    if case["kind"] == "adjoint":
        if case["method"] == "tree" or pairs * case["steps"] > 4e10:
            return None  # through a tree: the derivative of its frozen lists, not of the direct sum
        b = _bodies(case["scene"], n, _generator(seed))
        t = case["dt"] * case["steps"]
        target = torch.tensor((b.pos64() + t * b.vel64() + 1e-3).T.copy(), device="cuda")
        x, v, m = _state64(b)
        h, xs = 0.5 * case["dt"], [x.clone()]
        a, _ = _accel(x, m, eps)
        for _ in range(case["steps"]):
            v += h * a
            x = x + case["dt"] * v
            xs.append(x)
            a, _ = _accel(x, m, eps)
            v += h * a
        d = x - target
        loss = float((m * (d * d).sum(0)).sum())
        lx, lv, lm = 2 * m * d, torch.zeros_like(x), (d * d).sum(0)
        for s in range(case["steps"] - 1, -1, -1):
            lv += case["dt"] * lx
            gx, gm = _vjp(xs[s], m, (case["dt"] if s else h) * lv, eps)
            lx, lm = lx + gx, lm + gm
        return {"loss": loss, "gx": lx.T.cpu().numpy().copy(), "gv": lv.T.cpu().numpy().copy(), "gm": lm.cpu().numpy()}
    if pairs * (case["steps"] + 1) > 6e10:
        return None
    x, v, m = _state64(_bodies(case["scene"], n, _generator(seed)))
    a, _ = _accel(x, m, eps)
    for k in range(case["steps"]):
        v += 0.5 * case["dt"] * a
        x += case["dt"] * v
        a, phi = _accel(x, m, eps, phi=k == case["steps"] - 1)
        v += 0.5 * case["dt"] * a
    out = {}
    if case["log"] != "no":
        out = {"ke": 0.5 * float((m * (v * v).sum(0)).sum()), "pe": 0.5 * float((m * phi).sum())}
    if case["method"] == "tree":
        o = _morton_order(x)
        x, v, m = x[:, o], v[:, o], m[o]
    return out | _columns(x, v, m)


def _entries(n, theta):
    """About how long a body's interaction list is: 150 log2 n at theta 0.6, more below it."""
    return 150 * math.log2(max(n, 2)) * (0.6 / theta) ** 2


def work(case):
    """Bodies read and written once (32 bytes a body and direction); 20 operations a body pair, 35 a
    list entry of a tree (a third of them cells of 65); the adjoint four times the forward's."""
    if case["kind"] == "ensemble":
        # The mean over log-uniform sizes.
        u = (np.arange(1024) + 0.5) / 1024
        c = case["lo"] * (case["hi"] / case["lo"]) ** u
        per = np.where(c <= 8192, 20 * c * c, 35 * c * 150 * np.log2(c) * (0.6 / case["theta"]) ** 2)
        return {"bytes": 64.0 * case["systems"] * float(c.mean()),
                "flops": case["systems"] * case["steps"] * float(per.mean())}
    n = case["n"]
    per = 20.0 * n * n if case["method"] == "direct" else 35.0 * n * _entries(n, case["theta"])
    evals = {"steps": case.get("steps", 1), "forces": 1, "adjoint": 4 * case.get("steps", 1)}[case["kind"]]
    return {"bytes": 64.0 * n, "flops": per * evals}
