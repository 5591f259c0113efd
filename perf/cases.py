"""What the framework's users have it do, as cases that can be timed.

Each case is one pass through the public entry points (the Python binding of the C ABI):
segments of flat-histogram runs for each system and method, delayed-acceptance moves with
online training, and the surrogate's gradients and predictions on caller configurations.
A pass of a run continues the walkers' chains (or, where `fresh`, restarts them from their
uploaded configurations) and reads back what a program keeps of a segment: the ln w and
histogram planes, the energies and the configurations.

Sizes are those of the repository's own benchmark, tests and documented quickstart.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "sad-monte-carlo_gb300"))
import sadmc_gb300 as G  # noqa: E402

METHODS = {"sad": G.SAD, "samc": G.SAMC, "wl": G.WL}
CV_T = [0.25, 0.28, 0.30, 0.33, 0.36]


def listed():
    return [
        # The reference's own run: one 32x32 Ising walker, read back every 20 k moves.
        dict(name="ising32_one_walker", kind="ising", L=32, walkers=1, method="sad", moves=20000, lanes=0),
        # The same lattice as a batch of independent walkers, which is how a GPU runs it.
        dict(name="ising32_4096_walkers", kind="ising", L=32, walkers=4096, method="sad", moves=8192, lanes=0),
        # The headline workload end to end: fresh LJ31 walkers from host configurations,
        # descent, 1e8 moves, planes read back and the energies verified.
        dict(name="lj31_4096_fresh", kind="lj", n=31, radius=2.5, walkers=4096, method="sad", min_T=0.2,
             bin=0.134, e_lo=-134.268, moves=24414, lanes=0, fresh=True),
        # A segment of a converging LJ31 run followed by the per-walker heat capacities that
        # a convergence study looks at after each segment.
        dict(name="lj31_1024_segment_cv", kind="lj", n=31, radius=2.5, walkers=1024, method="sad", min_T=0.2,
             bin=0.134, e_lo=-134.268, moves=16384, lanes=0, fresh=False),
        # The 38-atom cluster with 8192 walkers, at the lanes per walker the autotuner picks
        # for it; the largest batch of the benchmark.
        dict(name="lj38_8192_segment", kind="lj", n=38, radius=3.5, walkers=8192, method="sad", min_T=0.05,
             bin=0.2, e_lo=-180.0, moves=8192, lanes=2, fresh=False),
        # Periodic WCA fluid, uneven N and density per walker, SAMC (autotuned lanes).
        dict(name="wca_2048_uneven", kind="wca", n_max=512, walkers=2048, method="samc", moves=2048, lanes=16),
        # Hard-core square well, N = 1024, Wang-Landau over contact counts (autotuned lanes).
        dict(name="square_well_1024", kind="sw", n=1024, walkers=1024, method="wl", moves=2048, lanes=32),
        # Delayed-acceptance moves whose surrogate collects and retrains during the run.
        dict(name="lj38_delayed_online", kind="da", n=38, radius=3.5, walkers=1024, moves=1024, collect=512,
             retrain=512, train_steps=20, batch=512),
        # One gradient evaluation of the surrogate on a minibatch of 512 LJ38 configurations.
        dict(name="surrogate_gradients_512", kind="grads", n=38, radius=3.5, configs=512),
        # Energies of a large set of configurations (screening or validation of a data set).
        dict(name="surrogate_predict_8192", kind="predict", n=38, radius=3.5, configs=8192),
        # Grand-canonical LJ cluster and WCA fluid, energy-number SAMC.
        dict(name="grand_lj31_4096", kind="grand_lj", n_max=31, radius=2.5, walkers=4096, moves=4096, lanes=0),
        dict(name="grand_wca200_512", kind="grand_wca", n_max=200, box=6.0, walkers=512, moves=4096, lanes=0),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["ising", "ising", "lj", "lj", "lj", "wca", "wca", "sw", "sw", "da", "grads", "predict",
                       "grand_lj", "grand_wca"])
    if kind == "ising":
        one = rng.random() < 0.4
        return dict(kind=kind, L=rng.randint(6, 36), walkers=1 if one else _log_int(rng, 2, 4096),
                    method=rng.choice(["sad", "sad", "wl", "samc"]), moves=_log_int(rng, 300, 16000), lanes=0)
    if kind == "lj":
        n = rng.choice([13, 19, 31, 31, 38, 55]) if rng.random() < 0.6 else rng.randint(8, 60)
        radius = round(0.62 * (n / 0.75) ** (1.0 / 3.0) + rng.uniform(0.5, 1.2), 3)
        return dict(kind=kind, n=n, radius=radius, walkers=_log_int(rng, 1, 6000),
                    method=rng.choice(["sad", "sad", "sad", "wl", "samc"]), min_T=round(rng.uniform(0.05, 0.3), 3),
                    bin=round(rng.uniform(0.1, 0.5), 3), e_lo=round(-5.5 * n, 1), moves=_log_int(rng, 500, 9000),
                    lanes=rng.choice([0, 0, 0, 1, 2, 8]), fresh=rng.random() < 0.5)
    if kind == "wca":
        return dict(kind=kind, n_max=rng.choice([64, 128, 256, 512]), walkers=_log_int(rng, 1, 2000),
                    method=rng.choice(["samc", "samc", "sad", "wl"]), moves=_log_int(rng, 200, 2000),
                    lanes=rng.choice([0, 16, 16, 32]))
    if kind == "sw":
        return dict(kind=kind, n=rng.randint(64, 1024), walkers=_log_int(rng, 1, 1000),
                    method=rng.choice(["wl", "wl", "sad", "samc"]), moves=_log_int(rng, 200, 2000),
                    lanes=rng.choice([0, 32, 32, 16]))
    if kind == "da":
        n = rng.randint(13, 50)
        return dict(kind=kind, n=n, radius=round(0.62 * (n / 0.75) ** (1.0 / 3.0) + 1.0, 3),
                    walkers=_log_int(rng, 32, 1000), moves=_log_int(rng, 256, 1024), collect=256,
                    retrain=rng.choice([256, 512]), train_steps=rng.randint(5, 20), batch=rng.randint(64, 512))
    if kind in ("grads", "predict"):
        n = rng.randint(8, 80)
        return dict(kind=kind, n=n, radius=round(0.62 * (n / 0.75) ** (1.0 / 3.0) + 1.0, 3),
                    configs=_log_int(rng, 1, 700 if kind == "grads" else 300000 // n))
    if kind == "grand_lj":
        return dict(kind=kind, n_max=rng.randint(8, 40), radius=round(rng.uniform(2.0, 3.0), 3),
                    walkers=_log_int(rng, 8, 4000), moves=_log_int(rng, 500, 4000), lanes=0)
    return dict(kind=kind, n_max=rng.randint(40, 200), box=round(rng.uniform(4.5, 6.5), 3),
                walkers=_log_int(rng, 4, 500), moves=_log_int(rng, 500, 4000), lanes=0)


# ---- inputs ---------------------------------------------------------------------------
def _clusters(count, n, radius, rng, dmin=0.8):
    """`count` clusters of n atoms uniform in the sphere, each atom redrawn while closer
    than dmin to an earlier one: [count, n, 3] float64."""
    out = np.full((count, n, 3), 1e3)
    for k in range(n):
        todo = np.arange(count)
        d = dmin
        for attempt in range(400):
            p = rng.uniform(-radius, radius, (len(todo), 3))
            ok = (p * p).sum(1) < radius * radius
            if k:
                ok &= ((out[todo, :k] - p[:, None, :]) ** 2).sum(2).min(1) >= d * d
            out[todo[ok], k] = p[ok]
            todo = todo[~ok]
            if not len(todo):
                break
            if attempt % 100 == 99:
                d *= 0.9
        else:
            raise ValueError("the sphere is too small for its atoms")
    return out


def _wca_boxes(walkers, n_max, rng):
    """Uneven N and density: random subsets of a jittered simple cubic lattice."""
    # the sizes in equal shares, in an order of the seed's
    ns = rng.permutation(np.resize([n for n in (512, 256, 128, 64) if n <= n_max], walkers))
    rhos = rng.uniform(0.6, 0.9, walkers)
    out = []
    for n, rho in zip(ns, rhos):
        edge = (n / rho) ** (1 / 3)
        m = int(np.ceil(n ** (1 / 3) - 1e-9))
        g = np.indices((m, m, m)).reshape(3, -1).T.astype(float)
        g = g[rng.permutation(len(g))[:n]]
        out.append((int(n), edge, np.mod((g + 0.5 + rng.uniform(-0.05, 0.05, g.shape)) * (edge / m), edge)))
    return out


def _sw_boxes(walkers, n, rng):
    """Hard spheres on a jittered FCC lattice, packing fraction uniform in [0.30, 0.50]."""
    m = int(np.ceil((n / 4) ** (1 / 3) - 1e-9))
    base = np.array([(0, 0, 0), (0.5, 0.5, 0), (0.5, 0, 0.5), (0, 0.5, 0.5)])
    sites = (np.indices((m, m, m)).reshape(3, -1).T.astype(float)[:, None, :] + base[None]).reshape(-1, 3)
    # sites that stay empty lower the densest packing that the lattice can hold
    top = min(0.50, 0.70 * n / len(sites))
    out = []
    for eta in rng.uniform(min(0.30, 0.6 * top), top, walkers):
        edge = (n * np.pi / (6 * eta)) ** (1 / 3)
        pick = sites[rng.permutation(len(sites))[:n]]
        out.append((n, edge, np.mod((pick + rng.uniform(-0.004, 0.004, pick.shape)) * (edge / m), edge)))
    return out


def _lj_energies(pos):
    """FP64 Lennard-Jones energies of [configs, n, 3]."""
    e = np.zeros(len(pos))
    n = pos.shape[1]
    for i in range(n - 1):
        s = 1.0 / ((pos[:, i + 1:] - pos[:, i:i + 1]) ** 2).sum(2)
        e += (4 * (s ** 6 - s ** 3)).sum(1)
    return e


_SHAPES = [(32, 64), (64,), (64, 64), (64,), (64,), (1,)]  # W1, b1, W2, b2, w3, b3


def _params(seed):
    """Surrogate weights N(0, 1/fan_in) with small biases, flat."""
    rng = np.random.default_rng(seed + 1)
    parts = [rng.normal(0, (1 / math.sqrt(sh[0]) if len(sh) == 2 or k == 4 else 0.05), sh)
             for k, sh in enumerate(_SHAPES)]
    return np.concatenate([np.ravel(q) for q in parts]).astype(np.float32)


def _surrogate_inputs(case, seed):
    """Configurations [configs, n, 3] and their target energies, binary32."""
    pos = _clusters(case["configs"], case["n"], case["radius"], np.random.default_rng(seed)).astype(np.float32)
    return pos, _lj_energies(pos.astype(np.float64)).astype(np.float32)


def _padded(a, shape):
    """A fixed-width record of an array whose extent grows with the run."""
    out = np.zeros(shape, a.dtype)
    out[tuple(slice(0, k) for k in a.shape)] = a
    return out


def _pinned(count, dtype):
    t = torch.empty(count, dtype=torch.float64 if dtype is np.float64 else torch.int64).pin_memory()
    a = t.numpy()
    return t, (a if dtype is np.float64 else a.view(np.uint64))


def _batch(case, seed):
    """The batch of a run and its host configurations."""
    rng = np.random.default_rng(seed)
    kind, W, method = case["kind"], case["walkers"], METHODS[case.get("method", "sad")]
    if kind == "ising":
        L = case["L"]
        cfg = G.make_config(G.ISING, W, L, method=method, min_T=0.2, t0=1e4, e_lo=-2.0 * L * L - 8,
                            e_hi=2.0 * L * L + 8, seed=seed, lanes_per_walker=case["lanes"])
        return G.Batch(cfg, [(L, 0.0, (0, 0, 0))] * W), np.where(rng.random(W * L * L) < 0.5, -1.0, 1.0), W * L * L
    if kind in ("lj", "da"):
        n, radius = case["n"], case["radius"]
        cfg = G.make_config(G.LJ, W, n, method=method, min_T=case.get("min_T", 0.05), t0=1e4,
                            energy_bin=case.get("bin", 0.2), max_allowed=0.0, e_lo=case.get("e_lo", -5.5 * n),
                            e_hi=1.0, target_rate=0.5, translation_scale=0.1, seed=seed,
                            lanes_per_walker=case.get("lanes", 0))
        conf = _clusters(W, n, radius, rng)
        return G.Batch(cfg, [(n, radius, (0, 0, 0))] * W), conf.reshape(-1), W * 3 * n
    if kind == "wca":
        boxes = _wca_boxes(W, case["n_max"], rng)
        cfg = G.make_config(G.WCA, W, max(b[0] for b in boxes), method=method, t0=1e4, energy_bin=1.0,
                            max_allowed=500.0, translation_scale=0.1, e_lo=-1.0, e_hi=501.0, seed=seed,
                            resum_interval=4096, lanes_per_walker=case["lanes"])
    else:
        n = case["n"]
        boxes = _sw_boxes(W, n, rng)
        cfg = G.make_config(G.SW, W, n, method=method, t0=1e4, well_width=1.3, translation_scale=0.05,
                            e_lo=-6.0 * n - 2, e_hi=2.0, seed=seed, lanes_per_walker=case["lanes"])
    b = G.Batch(cfg, [(n, 0.0, (edge, edge, edge)) for n, edge, _ in boxes])
    return b, np.concatenate([p.reshape(-1) for _, _, p in boxes]), sum(3 * n for n, _, _ in boxes)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("grads", "predict"):
        n, radius = case["n"], case["radius"]
        b = G.Batch(G.make_config(G.LJ, 1, n, energy_bin=0.2, max_allowed=0.0, e_lo=-5.5 * n, e_hi=1.0, seed=seed),
                    [(n, radius, (0, 0, 0))])
        b.surrogate_init(seed=seed, ring_capacity=64)
        b.surrogate_set_params(_params(seed))
        pos, target = _surrogate_inputs(case, seed)
        return dict(case=case, batch=b, pos=pos, target=target)
    if kind == "grand_lj":
        return dict(case=case, batch=G.GrandBatch(G.make_grand_config(
            case["walkers"], case["n_max"], case["radius"], method=G.SAMC, t0=1e4, energy_bin=0.5, max_allowed=10.0,
            translation_scale=0.1, addremove_probability=0.1, e_lo=-5.5 * case["n_max"], e_hi=12.0, seed=seed,
            lanes_per_walker=case["lanes"])))
    if kind == "grand_wca":
        return dict(case=case, batch=G.GrandBatch(G.make_grand_config(
            case["walkers"], case["n_max"], box=(case["box"],) * 3, method=G.SAMC, t0=1e4, energy_bin=1.0,
            max_allowed=400.0, translation_scale=0.1, addremove_probability=0.2, e_lo=-1.0, e_hi=402.0, seed=seed,
            lanes_per_walker=case["lanes"])))
    b, conf, values = _batch(case, seed)
    nb = b.plane_bins()
    s = dict(case=case, batch=b, lnw=_pinned(b.W * nb, np.float64), hist=_pinned(b.W * nb, np.uint64),
             state=_pinned(values, np.float64), conf=_pinned(values, np.float64))
    s["conf"][1][:] = conf
    if not case.get("fresh"):
        # a run under way: the walkers have found most of their bins
        b.upload(s["conf"][1])
        b.initialize()
        if kind == "da":
            b.surrogate_init(seed=seed, ring_capacity=65536)
            b.run_online(4096, False, collect_interval=512, retrain_interval=2048, train_steps=100, batch=512,
                         lr=2e-3, seed=seed)
        else:
            b.run({"ising": 200000 if b.W == 1 else 16384, "lj": 16384}.get(kind, 1024))
    return s


def _read(s):
    """A segment's results in the program's own host buffers."""
    b = s["batch"]
    lnw, hist, rng, mins = b.read_planes(s["lnw"][1], s["hist"][1])
    rc = G.lib().sadmc_read_state(b.h, 0, b.W, s["state"][1].ctypes.data_as(ctypes.c_void_p))
    if rc:
        raise RuntimeError(G.lib().sadmc_last_error().decode())
    return dict(lnw=lnw, hist=hist.view(np.int64), range=rng, bins_min=mins, state=s["state"][1],
                energy=b.energies())


def run(state):
    case, b = state["case"], state["batch"]
    kind = case["kind"]
    if kind == "grads":
        loss, grads = b.surrogate_loss_grads(state["pos"], state["target"])
        return dict(loss=loss, grads=grads)
    if kind == "predict":
        return dict(energy=b.surrogate_predict(state["pos"]))
    if kind.startswith("grand"):
        # a handle reads one walker at a time: a monitoring program looks at a few
        b.run(case["moves"])
        W, cfg = case["walkers"], b.cfg
        shape = (int(math.ceil((cfg.e_hi - cfg.e_lo) / cfg.energy_bin)) + 8, case["n_max"] + 1)
        out = {}
        for w in sorted({0, W // 3, W // 2, W - 1}):
            bins = b.bins(w)
            out["walker%d" % w] = dict(state=_padded(b.state(w), (case["n_max"], 3)),
                                       scalars=np.array(list(b.scalars(w).values())),
                                       lnw=_padded(bins["lnw"], shape),
                                       hist=_padded(bins["hist"], shape).view(np.int64),
                                       round_trips=_padded(bins["round_trips"], shape).view(np.int64))
        return out
    if kind == "da":
        stats = b.run_online(case["moves"], True, collect_interval=case["collect"], retrain_interval=case["retrain"],
                             train_steps=case["train_steps"], batch=case["batch"], lr=1e-3, seed=7)
        return dict(_read(state), stats=stats.view(np.int64), params=b.surrogate_params())
    if case.get("fresh"):
        b.upload(state["conf"][1])
        b.initialize()
        b.run(case["moves"])
        return dict(_read(state), verified=b.compute_energies())
    b.run(case["moves"])
    out = _read(state)
    if kind == "lj":
        out["cv"] = b.heat_capacities(CV_T)
    if b.W == 1:
        nb = b.plane_bins()
        out["bins"] = {k: _padded(v.view(np.int64) if v.dtype == np.uint64 else v, nb)
                       for k, v in b.bins(0).items() if isinstance(v, np.ndarray)}
        out["scalars"] = np.array(list(b.scalars(0).values()))
    return out


# ---- what a pass cannot do without ------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("grads", "predict"):
        rows = case["configs"] * case["n"]
        rbf = rows * (case["n"] - 1) * 32 * 5.0
        params = 6337 * 4
        if kind == "grads":
            return {"bytes": rows * 12.0 + case["configs"] * 4 + 2 * params, "flops": rows * 32768.0 + rbf}
        return {"bytes": rows * 12.0 + case["configs"] * 4 + params, "flops": rows * 12416.0 + rbf}
    moves = float(case["walkers"]) * case["moves"]
    if kind == "ising":
        bins = case["L"] ** 2 + 8
        # 4 neighbours, the flip's energy, the acceptance test and the weight update
        return {"bytes": case["walkers"] * (bins * 16.0 + case["L"] ** 2 * 8), "flops": moves * 12}
    if kind in ("lj", "da"):
        n = case["n"]
        bins = (1.0 - case.get("e_lo", -5.5 * n)) / case.get("bin", 0.2) + 5
        per = 30.0 * (n - 1)
        if kind == "da":
            per += 2.0 * n * 6208 + 2.0 * (n - 1) * 32 * 5
        return {"bytes": case["walkers"] * (bins * 16 + n * 24.0), "flops": moves * per}
    if kind == "wca":
        n = np.array([m for m in (64, 128, 256, 512) if m <= case["n_max"]], float)
        edge = (n / 0.75) ** (1 / 3)
        cand = 27 * n / np.floor(edge / 2 ** (1 / 6)) ** 3 - 1
        return {"bytes": case["walkers"] * (507 * 16.0 + float(n.mean()) * 24), "flops": moves * 30 * float(cand.mean())}
    if kind == "sw":
        n = case["n"]
        edge = (n * math.pi / (6 * 0.4)) ** (1 / 3)
        cand = 27 * n / max(3, math.floor(edge / 1.3)) ** 3 - 1
        return {"bytes": case["walkers"] * ((6.0 * n + 8) * 16 + n * 24), "flops": moves * 16 * cand}
    if kind == "grand_lj":
        return {"bytes": case["walkers"] * 24.0 * case["n_max"], "flops": moves * 30 * 0.4 * case["n_max"]}
    cells = math.floor(case["box"] / 2 ** (1 / 6)) ** 3
    return {"bytes": case["walkers"] * 24.0 * case["n_max"], "flops": moves * 30 * 27.0 * 20 / cells}


# ---- the surrogate in 64 bits -----------------------------------------------------------
def _silu(z):
    return z / (1.0 + np.exp(-z))


def _dsilu(z):
    s = 1.0 / (1.0 + np.exp(-z))
    return s * (1.0 + z * (1.0 - s))


def exact(case, seed):
    """The surrogate's loss, gradients and energies as FP64 numpy gives them for the same
    inputs.  The Markov chains have no such value: their decisions are on binary32 pair
    energies, and a run is what follows from all of them."""
    if case["kind"] not in ("grads", "predict"):
        return None
    flat, p, o = _params(seed).astype(np.float64), [], 0
    for shape in _SHAPES:
        k = int(np.prod(shape))
        p.append(flat[o:o + k].reshape(shape))
        o += k
    W1, b1, W2, b2, w3, b3 = p
    pos, target = _surrogate_inputs(case, seed)
    pos, target = pos.astype(np.float64), target.astype(np.float64)
    C, n = pos.shape[:2]
    centres = 0.8 + 2.2 * np.arange(32) / 31
    desc = np.empty((C, n, 32))
    for i in range(n):
        r = np.sqrt(((pos - pos[:, i:i + 1]) ** 2).sum(2))
        r[:, i] = np.inf
        for k in range(32):
            desc[:, i, k] = np.exp(-((r - centres[k]) ** 2) / (2 * 0.1 ** 2)).sum(1)
    x = desc.reshape(C * n, 32)
    z1 = x @ W1 + b1
    h1 = _silu(z1)
    z2 = h1 @ W2 + b2
    h2 = _silu(z2)
    e = (h2 @ w3 + b3[0]).reshape(C, n).sum(1)
    if case["kind"] == "predict":
        return dict(energy=e)
    res = e - target
    de = np.repeat(2 * res / C, n)
    d2 = de[:, None] * w3 * _dsilu(z2)
    d1 = (d2 @ W2.T) * _dsilu(z1)
    grads = [x.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0), h2.T @ de, np.array([de.sum()])]
    return dict(loss=float((res ** 2).mean()), grads=np.concatenate([np.ravel(q) for q in grads]))
