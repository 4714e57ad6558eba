"""Performance cases: what a program does with this library, through its public entry points.

A pass is one leg of a simulation: the colony's state goes up from pinned host arrays into an
engine that the program keeps, the engine makes the steps between two frames, and the state comes
back. The colonies are the benchmark's models (2D growth, the WCA configuration, the 3D channel, a
sweep of colonies in one handle) and the single-element cell-cycle model of the shipped runs, from
the first hundreds of cells of a run to the million-cell checkpoint. One case bins elements with
the entry point for callers that own their memory.

run() returns what the program reads back, in arrays of the colony's capacity (places past the cells
stay zero): positions, cycles and cell state as the engine holds them (FP64, int32). Velocities, pressures and forces come back in FP64 from the FP64 forms; the
mixed forms evaluate them in FP32, and what follows from them at once (the cycle activity rho, which
feels a contact's pressure from its first touch, and DPD's velocities) comes back in FP32, as
frames store it. The legs of the cell-cycle model are short: its motility follows the
velocity's direction, which amplifies last-bit differences by about 14 % per step.

exact() restates the models in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

import cil_cuda_gb300 as G
from cil_cuda_gb300 import skin_scheduler

NEVER = 2**30
SIGMA_1 = 1.1283791670955126  # diameter of a disk of unit area (SIGMA_CORE of the shipped runs)


def listed():
    return [
        # the early part of a growth run: a few hundred cells, every launch counts
        dict(name="growth_300_skin", kind="colony", model="growth", cells=300, precision="mixed", skin=1,
             integrator="euler", steps=100),
        # the first benchmark configuration at its size, in the parity form
        dict(name="wca_4096_fp64", kind="colony", model="wca", cells=4096, precision="fp64", skin=0,
             integrator="euler", steps=50),
        # a growth colony in the parity form, which rebuilds its bins every step
        dict(name="growth_250k_fp64", kind="colony", model="growth", cells=250001, precision="fp64", skin=0,
             integrator="euler", steps=10),
        # the mixed form without lists (a run description without SKIN), an odd size
        dict(name="growth_200k_mixed", kind="colony", model="growth", cells=200003, precision="mixed", skin=0,
             integrator="euler", steps=30),
        # the headline workload: the 1M-cell checkpoint, lists and learned scheduler, one frame
        dict(name="growth_1m_skin", kind="colony", model="growth", cells=1000000, precision="mixed", skin=1,
             integrator="euler", steps=100),
        # the 3D channel in the form it is run in
        dict(name="channel_400k_skin", kind="colony", model="channel", cells=400000, precision="mixed", skin=1,
             integrator="euler", steps=40),
        # the 3D channel in the parity form
        dict(name="channel_60k_fp64", kind="colony", model="channel", cells=60001, precision="fp64", skin=0,
             integrator="euler", steps=8),
        # a parameter sweep: colonies of log-uniform size in one handle
        dict(name="sweep_64", kind="sweep", colonies=64, cells_lo=500, cells_hi=16000, steps=300),
        # the shipped runs' early sizes: 1024 cells of the cell-cycle model
        dict(name="cycle_1k_fp64", kind="cycle", cells=1024, precision="fp64", integrator="euler", steps=50),
        # the cell-cycle model at a late size, FP64
        dict(name="cycle_1m_fp64", kind="cycle", cells=1000000, precision="fp64", integrator="euler", steps=10),
        # the DPD integrator with FP32 pair terms
        dict(name="dpd_150k_mixed", kind="cycle", cells=150000, precision="mixed", integrator="dpd", steps=12),
        # element binning for a host framework with its own device memory
        dict(name="bins_1m", kind="bins", elements=1000003, dim=2, per_bin=2.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["colony"] * 6 + ["cycle"] * 3 + ["sweep", "bins"])
    if kind == "colony":
        model = rng.choice(["growth", "growth", "wca", "channel"])
        precision = rng.choice(["fp64", "mixed", "mixed"])
        skin = rng.choice([0, 1, 1]) if precision == "mixed" else 0
        integrator = rng.choice(["euler", "euler", "euler", "heun"])
        hi = 800000 if skin else 250000
        hi = hi // 2 if model == "channel" else hi
        cells = _log_int(rng, 300 if model != "channel" else 3000, hi)
        slow = (6 if precision == "fp64" else 2 if not skin else 1) * (2 if integrator == "heun" else 1)
        return dict(kind=kind, model=model, cells=cells, precision=precision, skin=skin, integrator=integrator,
                    steps=max(5, min(100, rng.randint(30, 100) // slow)))
    if kind == "cycle":
        precision = rng.choice(["fp64", "mixed"])
        integrator = rng.choice(["euler", "euler", "dpd"])
        cells = _log_int(rng, 500, 600000 if integrator == "euler" or precision == "mixed" else 200000)
        return dict(kind=kind, cells=cells, precision=precision, integrator=integrator, steps=rng.randint(5, 10))
    if kind == "sweep":
        lo = _log_int(rng, 200, 2000)
        return dict(kind=kind, colonies=rng.randint(4, 64), cells_lo=lo, cells_hi=lo * rng.randint(2, 16),
                    steps=rng.randint(100, 300))
    return dict(kind=kind, elements=_log_int(rng, 1000, 1048576), dim=rng.choice([2, 3]),
                per_bin=round(rng.uniform(1.2, 6.0), 2))


# ---------------------------------------------------------------- inputs
def _params(dim, law, box, **over):
    p = dict(dim=dim, force_law=law, noise_per_cell=0, divide=0, box=list(box) + [0.0] * (3 - len(box)),
             periodic=[1] * dim + [0] * (3 - dim), nwalls=0, wall_dir=[1, -1], wall_pos=[0.0, 0.0], wall_E=0.0,
             epsilon=1.0, rcut_scale=1.0, zeta=[1.0, 1.0], motility=[0.0, 1.0], kappa=10.0, rest0=0.5, rest1=1.0,
             noise_D=0.01, dt=1e-4, div_tau_mu=1.0, div_tau_sigma=0.1, apop_rate=0.0, well_epsilon=0.0,
             well_sigma=0.0, force_shifted=0)
    p.update(over)
    return p


def _wrap(x, box, periodic):
    for d, L in enumerate(box):
        if periodic[d]:
            x[..., d] %= L
            x[..., d][x[..., d] >= L] = 0.0
    return x


def _ages(rng, n, p):
    """Cycles of a colony in steady growth: ages uniform over a drawn cycle length."""
    if not p["divide"]:
        return np.zeros(n, np.int32), np.full(n, NEVER, np.int32), np.full(n, p["rest0"])
    dt = p["dt"]
    span = np.maximum(np.rint(rng.normal(p["div_tau_mu"], p["div_tau_sigma"], n) / dt), 1).astype(np.int64)
    age = (rng.random(n) * span).astype(np.int64)
    rest = p["rest0"] + (p["rest1"] - p["rest0"]) * age / span
    return (-age).astype(np.int32), (span - age).astype(np.int32), rest


def _growth(rng, n, tau=1.0, motility=1.0):
    """A grown colony: cells uniform in a disk at packing fraction 0.8 of a periodic box."""
    sigma = np.clip(rng.normal(1.0, 0.1, (n, 2)), 0.7, 1.3)
    R = math.sqrt(float(np.sum(sigma**2)) / 4 / 0.8)
    L = max(2.6 * R, 12.0)
    p = _params(2, G.FORCE_SOFTCORE, [L, L], epsilon=5.0, divide=1, div_tau_mu=tau, div_tau_sigma=0.1 * tau,
                apop_rate=0.01 / tau, motility=[0.0, motility])
    t0, tsw, rest = _ages(rng, n, p)
    r, th, ax = R * np.sqrt(rng.random(n)), 2 * np.pi * rng.random(n), 2 * np.pi * rng.random(n)
    centre = np.stack([L / 2 + r * np.cos(th), L / 2 + r * np.sin(th)], axis=1)
    half = (0.5 * rest)[:, None] * np.stack([np.cos(ax), np.sin(ax)], axis=1)
    pos = _wrap(np.stack([centre - half, centre + half], axis=1), [L, L], [1, 1])
    return p, dict(pos=pos, sigma=sigma, t0=t0, tswitch=tsw)


def _wca(rng, n):
    """WCA cells at packing fraction 0.8, nearly aligned on a jittered lattice (no deep overlaps)."""
    nx = max(3, int(math.sqrt(n * 1.155 / 1.7)))
    ny = -(-n // nx)
    L = max(1.7 * nx, 1.155 * ny)
    sigma = np.clip(rng.normal(1.0, 0.05, (n, 2)), 0.85, 1.15)
    p = _params(2, G.FORCE_LJ_WCA, [L, L], rcut_scale=2 ** (1 / 6))
    t0, tsw, rest = _ages(rng, n, p)
    i = np.arange(n)
    centre = np.stack([(i % nx + 0.5) * L / nx, (i // nx + 0.5) * L / ny], axis=1) + rng.uniform(-0.03, 0.03, (n, 2))
    ax = rng.uniform(-0.1, 0.1, n)
    half = (0.5 * rest)[:, None] * np.stack([np.cos(ax), np.sin(ax)], axis=1)
    pos = _wrap(np.stack([centre - half, centre + half], axis=1), [L, L], [1, 1])
    return p, dict(pos=pos, sigma=sigma, t0=t0, tswitch=tsw)


def _channel(rng, n):
    """The 3D Hertzian channel between walls at z = 0 and 20, on a jittered lattice."""
    H = 20.0
    lxy = max(math.sqrt(n * 2.09 / (H - 1.5)), 8.0)
    sigma = rng.uniform(0.9, 1.1, (n, 2))
    p = _params(3, G.FORCE_HERTZ, [lxy, lxy, H], epsilon=100.0, divide=1, apop_rate=0.01, dt=5e-5, noise_D=0.005,
                periodic=[1, 1, 0], nwalls=2, wall_pos=[0.0, H], wall_E=100.0)
    t0, tsw, rest = _ages(rng, n, p)
    nz = 14
    nx = max(1, int(math.ceil(math.sqrt(n / nz))))
    i = np.arange(n)
    a = lxy / nx
    centre = np.stack([(i % nx + 0.5) * a, (i // nx % nx + 0.5) * a,
                       0.75 + (i // (nx * nx) + 0.5) * (H - 1.5) / nz], axis=1)
    centre[:, :2] += rng.uniform(-0.1, 0.1, (n, 2)) * a
    ax = rng.normal(size=(n, 3))
    ax /= np.linalg.norm(ax, axis=1, keepdims=True)
    half = (0.5 * rest)[:, None] * ax
    pos = _wrap(np.stack([centre - half, centre + half], axis=1), [lxy, lxy, H], [1, 1, 0])
    pos[..., 2] = np.clip(pos[..., 2], 0.5, H - 0.5)
    return p, dict(pos=pos, sigma=sigma, t0=t0, tswitch=tsw)


_MODELS = {"growth": _growth, "wca": _wca, "channel": _channel}


def _cycle(rng, n, case):
    """The single-element model of the shipped 2D runs, which grow one island of cells in a periodic
    box: Hertz contacts with adhesion, motility 1, a jittered square lattice of spacing 1.1, cycle
    phases uniform."""
    side = max(4, int(math.ceil(math.sqrt(n))))
    L = 1.25 * side + 4.0
    i = np.arange(n)
    pos = np.stack([(i % side) * 1.1, (i // side) * 1.1], axis=1) + 0.5 * (L - 1.1 * side + 1.1)
    pos += rng.uniform(-0.05, 0.05, (n, 2))
    p = dict(box=[L, L, 0.0], dt=1e-5, motility=1.0, zeta=0.01, v1=15.0,
             precision=1 if case["precision"] == "mixed" else 0)
    if case["integrator"] == "dpd":
        p.update(integrator=G.CYCLE_DPD, mass=1.0, kbt=0.003, dis_diff=1.0, dis_bg=0.01)
    return p, dict(pos=pos, sigma=np.full(n, SIGMA_1), theta=rng.random(n), rho=np.ones(n), angvel=np.full(n, 1e-5))


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 7])
    if case["kind"] == "colony":
        return _MODELS[case["model"]](rng, case["cells"])
    if case["kind"] == "sweep":
        out, ratio = [], case["cells_hi"] / case["cells_lo"]
        for c in range(case["colonies"]):
            n = int(case["cells_lo"] * ratio ** (c / max(1, case["colonies"] - 1)))
            tau = math.exp(rng.uniform(math.log(0.3), math.log(3.0)))
            out.append(_growth(rng, n, tau, float(rng.uniform(0.1, 2.0))))
        return out
    if case["kind"] == "cycle":
        return _cycle(rng, case["cells"], case)
    n, dim = case["elements"], case["dim"]
    L = (n / case["per_bin"]) ** (1.0 / dim) * 1.3
    return [L] * dim, rng.random((n, dim)) * L


def _capacity(n):
    return int(1.2 * n) + 64


def _pinned(shape, dtype=np.float64):
    t = {np.float64: torch.float64, np.int32: torch.int32}[dtype]
    return torch.zeros(shape, dtype=t, pin_memory=torch.cuda.is_available()).numpy()


def _pin(a, dtype):
    b = _pinned(a.shape, dtype)
    b[...] = a
    return b


# ---------------------------------------------------------------- the program's state
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("colony", "sweep"):
        colonies = [_inputs(case, seed)] if kind == "colony" else _inputs(case, seed)
        mixed = kind == "sweep" or case["precision"] == "mixed"
        lists = kind == "sweep" or case["skin"]
        skin = skin_scheduler.load()[2] if lists else 0.0
        heun = kind == "colony" and case["integrator"] == "heun"
        caps = [_capacity(len(s["sigma"])) for _, s in colonies]
        eng = G.Engine([p for p, _ in colonies], caps, precision=G.PREC_MIXED if mixed else G.PREC_FP64,
                       rng=G.RNG_PHILOX, seed=seed & 0xffffffff, skin=skin,
                       integrator=G.INTEGRATOR_HEUN if heun else G.INTEGRATOR_EULER)
        if lists:
            skin_scheduler.install(eng)
        types = dict(pos=np.float64, sigma=np.float64, t0=np.int32, tswitch=np.int32)
        ups = [{k: _pin(s[k], t) for k, t in types.items()} for _, s in colonies]
        cap, D = sum(caps), eng.dim
        out = dict(pos=_pinned((cap, 2, D)), sigma=_pinned((cap, 2)), t0=_pinned((cap,), np.int32),
                   tswitch=_pinned((cap,), np.int32))
        if not mixed:
            out["vel"] = _pinned((cap, 2, D))
        off = np.concatenate([[0], np.cumsum(caps)])
        views = [{k: v[off[c]:off[c + 1]] for k, v in out.items()} for c in range(len(caps))]
        return dict(case=case, engine=eng, ups=ups, out=out, views=views)
    if kind == "cycle":
        p, s = _inputs(case, seed)
        n = len(s["sigma"])
        cap = _capacity(n)
        eng = G.CycleEngine(p, cap, seed=seed & 0xffffffff)
        names, vecs = ["sigma", "sigma_t", "theta", "rho"], ["pos"]
        if case["precision"] == "fp64":
            names.append("pressure")
            vecs += ["vel", "force"]
        elif case["integrator"] == "dpd":
            vecs.append("vel")
        out = {k: _pinned((cap,)) for k in names}
        out.update({k: _pinned((cap, 2)) for k in vecs})
        view = G.CycleView(ncells=0, capacity=cap, **{k: G._dp(v) for k, v in out.items()})
        return dict(case=case, engine=eng, up={k: _pin(v, np.float64) for k, v in s.items()}, out=out, view=view)
    box, pos = _inputs(case, seed)
    n, dim = pos.shape
    nbins = 1
    for L in box:
        nbins *= max(1, int(L / 1.3))
    return dict(case=case, box=np.array(box), ns=np.zeros(3, np.int32), nbins=nbins,
                pos=torch.from_numpy(pos).cuda(), start=torch.zeros(nbins + 1, dtype=torch.int32, device="cuda"),
                elems=torch.zeros(n, dtype=torch.int32, device="cuda"))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("colony", "sweep"):
        eng, n = state["engine"], []
        for c, up in enumerate(state["ups"]):
            eng.upload(c, **up)
        eng.step(case["steps"])
        for c, view in enumerate(state["views"]):
            n.append(eng.download(c, want=(), out=view)["ncells"])
        return dict(state["out"], ncells=np.array(n))
    if kind == "cycle":
        eng, view, out = state["engine"], state["view"], state["out"]
        eng.upload(**state["up"])
        eng.step(case["steps"])
        eng._check(G.lib().cil_cycle_download(eng.h, view))
        res = dict(out, ncells=view.ncells)
        if case["precision"] == "mixed":
            for k in ("rho", "vel"):
                if k in res:
                    res[k] = res[k].astype(np.float32)
        return res
    st = G.lib().cil_bin_elements_noalloc(
        state["pos"].data_ptr(), len(state["elems"]), case["dim"], G._dp(state["box"]), 1.3, G._ip(state["ns"]),
        state["start"].data_ptr(), state["elems"].data_ptr(), state["nbins"], None)
    if st != 0:
        raise G.CilError(st, "cil_bin_elements_noalloc")
    return dict(start=state["start"], elems=state["elems"])


def work(case):
    """Per step: each element's position read and written, its diameter and id read, and its
    contacts' and own terms evaluated once per cell; once: the state up and down."""
    kind = case["kind"]
    if kind == "bins":
        n = case["elements"]
        return dict(bytes=n * (8 * case["dim"] + 4) + 4 * n / case["per_bin"], flops=2 * n * case["dim"])
    if kind == "cycle":
        n, s = case["cells"], case["steps"]
        per = 2 * 16 + 16 + 4 * 16 + 8  # position, velocity (written), sigma, sigma_t, theta, rho, speed
        dpd = case["integrator"] == "dpd"
        return dict(bytes=n * (s * (per + (48 if dpd else 0)) + 6 * 8 + 9 * 8),
                    flops=n * s * (120 + 5 * 40 + (5 * 60 if dpd else 0)))
    if kind == "sweep":
        D, s = 2, case["steps"]
        lo, hi = case["cells_lo"], case["cells_hi"]
        n = case["colonies"] * (hi - lo) / math.log(hi / lo)
        mixed = True
    else:
        D, s, n = (3 if case["model"] == "channel" else 2), case["steps"], case["cells"]
        s *= 2 if case["integrator"] == "heun" else 1
        mixed = case["precision"] == "mixed"
    e = 2 * n
    return dict(bytes=e * (s * (16 * D + (4 if mixed else 8) + 4) + 2 * (8 * D + 8 + 4)),
                flops=e * s * (60 + (4 if D == 2 else 6) * 20))


# ---------------------------------------------------------------- the models in 64 bits
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) of int64 tensors that hold 32-bit words."""
    m = 0xffffffff
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & m) ^ c1 ^ k0, p1 & m, ((p0 >> 32) & m) ^ c3 ^ k1, p0 & m
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c0, c1, c2, c3


def _block(c0, c1, c2, c3, seed):
    t = [v if torch.is_tensor(v) else torch.full_like(c0, v) for v in (c1, c2, c3)]
    return _philox(c0, t[0], t[1], t[2], seed & 0xffffffff, 0)


def _u24(w):
    return (w >> 8).double() * 2.0**-24


def _u53(a, b):
    return (((a << 21) ^ (b >> 11)) & ((1 << 53) - 1)).double() * 2.0**-53


def _normals24(a, b):
    r = torch.sqrt(-2.0 * torch.log(_u24(a) + 2.0**-24))
    t = 2 * math.pi * _u24(b)
    return r * torch.cos(t), r * torch.sin(t)


def _normals53(w):
    r = torch.sqrt(-2.0 * torch.log(1.0 - _u53(w[0], w[1])))
    t = 2 * math.pi * _u53(w[2], w[3])
    return r * torch.cos(t), r * torch.sin(t)


def _pairs(x, reach, box, periodic, near):
    """Calls near(i, j, d, r2) for the pairs with |d| < reach, d = x_j - x_i at the nearest image; an i
    comes at most once in a call."""
    n, D = x.shape
    dev = x.device
    L = torch.tensor(box[:D], dtype=torch.float64, device=dev)
    per = torch.tensor([bool(v) for v in periodic[:D]], device=dev)
    ns = [max(1, int(box[d] / reach)) for d in range(D)]
    ns = [v if v >= 3 else 1 for v in ns]
    b = torch.zeros(n, dtype=torch.int64, device=dev)
    co = []
    for d in range(D):
        v = (x[:, d] * (ns[d] / box[d])).long().clamp(0, ns[d] - 1)
        co.append(v)
        b = b * ns[d] + v
    order = torch.argsort(b)
    nb = math.prod(ns)
    count = torch.bincount(b, minlength=nb)
    end = torch.cumsum(count, 0)
    start = end - count
    most = int(count.max())
    every = torch.arange(n, device=dev)
    spans = [(-1, 0, 1) if ns[d] > 1 else (0,) for d in range(D)]
    for o in np.stack(np.meshgrid(*spans, indexing="ij"), -1).reshape(-1, D):
        ok = torch.ones(n, dtype=torch.bool, device=dev)
        t = torch.zeros_like(b)
        for d in range(D):
            v = co[d] + int(o[d])
            if not periodic[d]:
                ok &= (v >= 0) & (v < ns[d])
            t = t * ns[d] + v % ns[d]
        s, e = start[t], torch.where(ok, end[t], start[t])
        for k in range(most):
            i = every[s + k < e]
            if not len(i):
                break
            j = order[s[i] + k]
            d = x[j] - x[i]
            d = torch.where(per, d - torch.round(d / L) * L, d)
            r2 = (d * d).sum(1)
            sel = (r2 < reach * reach) & (i != j)
            near(i[sel], j[sel], d[sel], r2[sel])


def _colony_forces(p, x, sig, t0, tsw, ts, noise_at, seed):
    n, _, D = x.shape
    box, per = p["box"], p["periodic"]
    F = torch.zeros_like(x)
    r = x[:, 1] - x[:, 0]
    for d in range(D):
        if per[d]:
            r[:, d] -= torch.round(r[:, d] / box[d]) * box[d]
    ln = r.norm(dim=1, keepdim=True)
    rest = torch.full((n, 1), p["rest0"], dtype=torch.float64, device=x.device)
    if p["divide"]:
        frac = ((ts - t0).double() / (tsw - t0).double()).clamp(0, 1)
        rest = rest + (p["rest1"] - p["rest0"]) * frac[:, None]
    sp = p["kappa"] * (ln - rest)
    F[:, 0] = (sp - p["motility"][0]) * r / ln
    F[:, 1] = (p["motility"][1] - sp) * r / ln
    for w in range(p["nwalls"]):
        delta = (0.5 * sig - p["wall_dir"][w] * (x[..., D - 1] - p["wall_pos"][w])).clamp(min=0)
        F[..., D - 1] += p["wall_dir"][w] * p["wall_E"] * delta**1.5
    amp = math.sqrt(2 * p["noise_D"] / p["dt"])
    cell = torch.arange(n, device=x.device)
    if D == 2:
        w = _block(cell, noise_at, 1, 1, seed)
        for j in range(2):
            F[:, j] += p["zeta"][j] * amp * torch.stack(_normals24(w[2 * j], w[2 * j + 1]), 1)
    else:
        for j in range(2):
            w = _block(2 * cell + j, noise_at, 1, 0, seed)
            z = _normals24(w[0], w[1]) + _normals24(w[2], w[3])
            F[:, j] += p["zeta"][j] * amp * torch.stack(z[:3], 1)
    Fe, s = F.reshape(2 * n, D), sig.reshape(2 * n)
    law, eps, rcs = p["force_law"], p["epsilon"], p["rcut_scale"]

    def near(i, j, d, r2):
        rc = rcs * 0.5 * (s[i] + s[j])
        ok = ((i // 2) != (j // 2)) & (r2 < rc * rc)
        i, d, r2, rc = i[ok], d[ok], r2[ok], rc[ok]
        q = r2.sqrt()
        if law == G.FORCE_SOFTCORE:
            f = -eps * (1 - q / rc) ** 2 / q
        elif law == G.FORCE_HERTZ:
            f = -eps * (rc / rcs - q) ** 1.5 / q
        else:
            s6 = (rc * rc / (rcs * rcs) / r2) ** 3
            f = 24 * eps * (s6 - 2 * s6 * s6) / r2
        Fe[i] += f[:, None] * d

    _pairs(x.reshape(2 * n, D), rcs * float(s.max()), box, per, near)
    return F


def _whole(out, cells):
    """The cells' values in arrays of the colony's capacity; no value for whole numbers."""
    whole = {"ncells": None}
    for k, v in out.items():
        if v is not None:
            a = np.zeros((_capacity(cells),) + tuple(v.shape[1:]))
            a[:len(v)] = v.cpu().numpy()
            v = a
        whole[k] = v
    return whole


def _exact_colony(case, seed):
    p, st = _inputs(case, seed)
    D, dev = p["dim"], _dev()
    x, sig = (torch.from_numpy(st[k]).to(dev) for k in ("pos", "sigma"))
    t0, tsw = (torch.from_numpy(st[k]).long().to(dev) for k in ("t0", "tswitch"))
    heun = case["integrator"] == "heun"
    zeta = torch.tensor(p["zeta"], dtype=torch.float64, device=dev)[None, :, None]
    seed &= 0xffffffff
    vel = torch.zeros_like(x)

    def wrap(y):
        for d in range(D):
            if p["periodic"][d]:
                y[..., d] = torch.remainder(y[..., d], p["box"][d])
        return y

    for ts in range(case["steps"]):
        vel = torch.zeros_like(x)
        for half in range(2 if heun else 1):
            F = _colony_forces(p, x, sig, t0, tsw, ts, 2 * ts + half if heun else ts, seed)
            x = wrap(x + F / zeta * (p["dt"] / 2 if heun else p["dt"]))
            vel += F / zeta * (0.5 if heun else 1.0)
        now = ts + 1
        if p["divide"]:
            m = torch.nonzero(tsw == now)[:, 0]
            a, b = _block(m, now, 2, 0, seed), _block(m, now, 3, 0, seed)
            if D == 2:
                dirs = [torch.stack([torch.cos(2 * math.pi * _u24(w)), torch.sin(2 * math.pi * _u24(w))], 1)
                        for w in a[:2]]
            else:
                dirs = []
                for w, u in ((a[0], a[2]), (a[1], a[3])):
                    z, th = 2 * _u24(w) - 1, 2 * math.pi * _u24(u)
                    q = (1 - z * z).clamp(min=0).sqrt()
                    dirs.append(torch.stack([q * torch.cos(th), q * torch.sin(th), z], 1))
            rad = 0.5 * p["rest0"]
            back, front = x[m, 0].clone(), x[m, 1].clone()
            x[m] = wrap(torch.stack([front - rad * dirs[0], front + rad * dirs[0]], 1))
            x = torch.cat([x, wrap(torch.stack([back + rad * dirs[1], back - rad * dirs[1]], 1))])
            spans = [torch.round(p["div_tau_mu"] / p["dt"] + p["div_tau_sigma"] / p["dt"] * z).long().clamp(min=1)
                     for z in _normals24(b[0], b[1])]
            sig = torch.cat([sig, sig[m]])
            vel[m] = 0
            vel = torch.cat([vel, torch.zeros_like(x[len(vel):])])
            t0[m] = now
            tsw[m] = now + spans[1]
            t0, tsw = torch.cat([t0, t0[m]]), torch.cat([tsw, now + spans[0]])
        if p["apop_rate"] > 0:
            n, prob = len(x), p["apop_rate"] * p["dt"]
            if n * prob >= 30:
                return None
            w = _block(torch.zeros(1, dtype=torch.int64), now, 4, 0, seed)
            u, k = float(_u24(w[0])), 0
            pk = math.exp(n * math.log1p(-prob))
            cdf = pk
            while u > cdf and k < min(n, 200):
                pk *= (n - k) / (k + 1) * prob / (1 - prob)
                cdf += pk
                k += 1
            if k:
                w = _block(torch.arange(k), now, 5, 0, seed)
                gone = sorted(min(int(v * n), n - 1) for v in _u53(w[0], w[1]).tolist())
                if len(set(gone)) < k or k > 32:
                    return None  # picks drawn again: not restated
                keep = [c for c in range(n - k, n) if c not in gone]
                for hole, c in zip(gone, keep):
                    x[hole], sig[hole], vel[hole], t0[hole], tsw[hole] = x[c], sig[c], vel[c], t0[c], tsw[c]
                x, sig, vel, t0, tsw = (v[:n - k] for v in (x, sig, vel, t0, tsw))
    out = dict(pos=x, sigma=sig, t0=None, tswitch=None)
    if case["precision"] == "fp64":
        out["vel"] = vel
    return _whole(out, case["cells"])


def _exact_cycle(case, seed):
    q, st = _inputs(case, seed)
    dev, box, dt = _dev(), q["box"], q["dt"]
    S = {k: torch.from_numpy(v).to(dev) for k, v in st.items()}
    x, sig, th, rho, om = (S[k].clone() for k in ("pos", "sigma", "theta", "rho", "angvel"))
    sigt, v = sig.clone(), torch.zeros_like(x)
    dpd = case["integrator"] == "dpd"
    seed &= 0xffffffff
    E, nu, adh, p0, vs = 100.0, 0.5, 0.2, 5.0, math.pi * (SIGMA_1 / 2) ** 2
    c2, tau = 2 * (1 - nu * nu) / E, 1.0 / dt
    gam = q.get("dis_diff", 0.0)
    L = box[0]

    def contacts(key):
        n = len(x)
        cell = torch.arange(n, device=dev)
        w = _block(cell, key, 12, 0, seed)
        a = 2 * math.pi * _u53(w[0], w[1])
        vl = v.norm(dim=1, keepdim=True)
        u = torch.where(vl > 0, v / vl, torch.stack([torch.cos(a), torch.sin(a)], 1))
        F, pr = q["motility"] * u, torch.zeros(n, dtype=torch.float64, device=dev)

        def near(i, j, d, r2):
            ok = r2 <= (0.5 * (sig[i] + sig[j])) ** 2
            i, j, d, r = i[ok], j[ok], d[ok], r2[ok].sqrt()
            h = (0.5 * (sig[i] + sig[j]) - r).clamp(min=0)
            ra, rb = 0.5 * sig[torch.minimum(i, j)], 0.5 * sig[torch.maximum(i, j)]
            g = ra - (2 * rb * h - h * h) / (2 * (ra + rb - h))
            A = 2 * torch.sqrt(ra * ra - g * g)
            A = torch.where(torch.isnan(A), 2 * torch.minimum(ra, rb), A)
            f = -(h**1.5) / (0.75 * c2 * torch.sqrt(1 / ra + 1 / rb)) + adh * A
            pr[i] -= torch.where(A != 0, f / A, torch.zeros_like(f))
            F[i] += f[:, None] * d

        _pairs(x, float(sig.max()), box, [1, 1], near)
        return F, pr

    def pair_terms(key):
        Fd, Fr = torch.zeros_like(x), torch.zeros_like(x)
        sr = math.sqrt(2 * gam * q["kbt"])

        def near(i, j, d, r2):
            lo, hi = torch.minimum(i, j), torch.maximum(i, j)
            ok = r2.sqrt() < sig[lo]
            i, j, d, r, lo, hi = i[ok], j[ok], d[ok], r2[ok].sqrt(), lo[ok], hi[ok]
            w = (1 - r / sig[lo])[:, None]
            nd = d / r[:, None]
            z = torch.stack(_normals53(_block(lo, key, 16, hi, seed)), 1)
            Fd[i] -= gam * w * (v[i] - v[j]) * nd * nd
            Fr[i] += sr * w.sqrt() * nd * z

        _pairs(x, float(sig.max()), box, [1, 1], near)
        return Fd, Fr

    def dissipation():
        Fd = -q["dis_bg"] * v

        def near(i, j, d, r2):
            w = (1 - r2 / SIGMA_1)[:, None]
            nd2 = d * d / r2[:, None]
            Fd[i] -= gam * w * (v[i] - v[j]) * nd2

        _pairs(x, SIGMA_1, box, [1, 1], near)
        return Fd

    def kick():
        return v + (Fc * dt + Fd * dt + Fr * math.sqrt(dt)) / (4 * q["mass"])

    if dpd:
        (Fc, pr), (Fd, Fr) = contacts(0), pair_terms(0)
    for ts in range(case["steps"]):
        now = ts + 1
        if dpd:
            v = kick()
            x = torch.remainder(x + dt * v, L)
            (Fc, pr), (Fd, Fr) = contacts(now), pair_terms(now)
            v = kick()
            Fd = dissipation()
        else:
            F, pr = contacts(ts)
            v = F / (q["zeta"] * math.pi * (sig / 2) ** 2)[:, None]
            x = torch.remainder(x + dt * v, L)
        pn = pr.clamp(min=0) / p0
        th = th + om * rho.clamp(max=1.0)
        vt = math.pi * (sigt / 2) ** 2
        vt = vt + ((om * math.log(2) + (q["v1"] - 1) / tau) * rho - (vt - vs) / vs / tau) * vt
        sigt = 2 * torch.sqrt(vt / math.pi)
        sig = sigt.clone()  # CYCLE_TAU_P 0: the target is taken at once
        rn = 1 - rho - pn
        rho = rho + rn / tau * rho
        m = torch.nonzero(th >= 1)[:, 0]
        if len(m):
            w = [_block(m, now, 13, k, seed) for k in range(3)]
            new = sig[m] / math.sqrt(2.0)
            a = 2 * math.pi * _u53(w[0][0], w[0][1])
            dr = ((sig[m] - new) / 2)[:, None] * torch.stack([torch.sin(a), torch.cos(a)], 1)
            mu2, s2 = math.log(1 / math.sqrt(1.01)), math.sqrt(math.log(1.01))
            sp = [1.0 / torch.floor(torch.exp(mu2 + s2 * z) / dt + 0.5).clamp(min=1) for z in _normals53(w[2])]
            x = torch.cat([x, torch.remainder(x[m] + dr, L)])
            x[m] = torch.remainder(x[m] - dr, L)
            om[m] = sp[0]
            om = torch.cat([om, sp[1]])
            sig[m] = sigt[m] = new
            th[m] = 0
            v[m] = 0
            sig, sigt, th, rho, pr = (torch.cat([y, y[m]]) for y in (sig, sigt, th, rho, pr))
            v = torch.cat([v, v[m]])
            if dpd:
                for f in (Fc, Fd, Fr):
                    f[m] = 0
                Fc, Fd, Fr = (torch.cat([f, f[m]]) for f in (Fc, Fd, Fr))
    if not dpd:
        Fc, pr = contacts(case["steps"])
    out = dict(sigma=sig, sigma_t=sigt, theta=th, rho=rho, pos=x)
    if case["precision"] == "fp64" or dpd:
        out["vel"] = v
    if case["precision"] == "fp64":
        out.update(pressure=pr, force=Fc)
    return _whole(out, case["cells"])


def exact(case, seed):
    if case["kind"] == "colony":
        return _exact_colony(case, seed)
    if case["kind"] == "cycle":
        return _exact_cycle(case, seed)
    return None  # a sweep takes too long one colony at a time; bins are whole numbers
