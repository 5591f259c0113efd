"""The lean path of the bookkeeping (an ordinary move decided on binary32 thresholds) against
the FP64 oracle, where its thresholds matter: bins too narrow for it, energy bounds on either
side or none, every method, ragged batches and launches that end inside a table batch."""
import numpy as np
import pytest
from test_gpu_grand import SAME

from helpers import METHOD_KW, assert_bins_equal, assert_scalars_equal, ising_spins, lj_configs

pytestmark = pytest.mark.gpu

REPLAY_REL = 2e-5  # binary32 pair energies against FP64 ones, see test_gpu_lj.py


@pytest.mark.parametrize("lanes", [8, 2, 1])
@pytest.mark.parametrize("kw", [
    dict(method="sad", energy_bin=0.0001, min_allowed=-11.0, max_allowed=-10.0, e_lo=-13.0,
         e_hi=-8.0),                                                   # narrower than the estimate's error
    dict(method="sad", energy_bin=0.5, min_allowed=-25.0, max_allowed=-8.0),
    dict(method="sad", energy_bin=0.2, max_allowed=None, e_hi=400.0),  # no upper bound: proposals out of range
    dict(method="samc", energy_bin=0.2),
    dict(method="wl", energy_bin=2.0),
    dict(method="inv_t_wl", energy_bin=4.0),
    dict(method="canonical", energy_bin=0.2),
], ids=lambda k: f"{k['method']}-{k['energy_bin']}")
def test_lj_lean_path(gpu, oracle, kw, lanes):
    n, W, radius, seed, runs = 13, 5, 2.2, 11, (1200, 37, 500)
    okw = dict(METHOD_KW[kw["method"]], energy_bin=kw["energy_bin"], target_rate=0.5, translation_scale=0.1,
               max_allowed=kw.get("max_allowed", 0.0), min_allowed=kw.get("min_allowed"))
    okw = {k: v for k, v in okw.items() if v is not None}
    confs = lj_configs(oracle, n, radius, range(40, 40 + W))
    b = gpu.Batch(gpu.make_config(gpu.LJ, W, n, e_lo=kw.get("e_lo", -50.0), e_hi=kw.get("e_hi", 5.0), seed=seed,
                                  lanes_per_walker=lanes, **okw), [(n, radius, (0, 0, 0))] * W)
    b.upload(confs)
    b.initialize()
    E0 = b.energies()
    moves = sum(runs)
    b.set_trace(moves)
    for k in runs:
        b.run(k)
    out_of_range = b.status() & gpu.ST_BIN_RANGE
    for w in (0, 3, W - 1):
        if out_of_range[w]:
            continue  # the reference would have grown its bins
        e1, e2 = b.trace(w, moves)
        ow = oracle.Walker(oracle.make_config(oracle.LJ, n, radius=radius, seed=seed, walker=w, e0=float(E0[w]),
                                              **okw), confs[w])
        disc, mismatch = ow.run_override(e1, e2)
        assert mismatch == 0 and disc < REPLAY_REL, (w, mismatch, disc)
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_allclose(b.state(w), ow.state(), atol=1e-11)


@pytest.mark.parametrize("method,energy_bin,bounds", [
    ("sad", 1.0, None), ("sad", 3.0, (-300.0, 250.0)), ("sad", 0.25, (-60.0, 60.0)), ("samc", 8.0, (-400.0, None)),
    ("wl", 16.0, None), ("inv_t_wl", 16.0, (-450.0, 100.0)), ("canonical", 4.0, None)])
def test_ising_lean_path_bit_exact(gpu, oracle, method, energy_bin, bounds):
    L, W, seed = 16, 35, 13
    N = L * L
    kw = dict(METHOD_KW[method], energy_bin=energy_bin)
    if bounds:
        kw.update({k: v for k, v in zip(("min_allowed", "max_allowed"), bounds) if v is not None})
    b = gpu.Batch(gpu.make_config(gpu.ISING, W, L, e_lo=-2.0 * N - 20, e_hi=2.0 * N + 20, seed=seed,
                                  lanes_per_walker=1, **kw), [(L, 0.0, (0, 0, 0))] * W)
    spins = [ising_spins(L, 500 + w) for w in range(W)]
    b.upload(spins)
    b.initialize()
    for k in (7001, 33, 5000):
        b.run(k)
    for w in (0, 1, 31, 32, 34):
        ow = oracle.Walker(oracle.make_config(oracle.ISING, L, seed=seed, walker=w, **kw), spins[w])
        ow.run(12034)
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
    assert not b.status().any()


# An odd lattice has its energies on the bin edges, where the integer thresholds decide; one
# walker runs its chain with the planes in shared memory.
@pytest.mark.parametrize("method,L,W,energy_bin,bounds", [
    ("sad", 15, 33, 1.0, None), ("samc", 9, 3, 4.0, (-101.0, 60.0)), ("wl", 15, 33, 8.0, None),
    ("sad", 15, 3, 3.0, None), ("samc", 15, 1, 4.0, None), ("wl", 15, 1, 8.0, (-300.0, 200.0)),
    ("inv_t_wl", 16, 1, 8.0, None), ("samc", 16, 1, 0.5, (-202.0, 98.0))])
def test_ising_integer_thresholds(gpu, oracle, method, L, W, energy_bin, bounds):
    N, seed = L * L, 17
    kw = dict(METHOD_KW[method], energy_bin=energy_bin)
    if bounds:
        kw.update(min_allowed=bounds[0], max_allowed=bounds[1])
    b = gpu.Batch(gpu.make_config(gpu.ISING, W, L, e_lo=-2.0 * N - 20, e_hi=2.0 * N + 20, seed=seed, **kw),
                  [(L, 0.0, (0, 0, 0))] * W)
    spins = [ising_spins(L, 700 + w) for w in range(W)]
    b.upload(spins)
    b.initialize()
    for k in (7001, 33, 5000):
        b.run(k)
    for w in {0, W // 2, W - 1}:
        ow = oracle.Walker(oracle.make_config(oracle.ISING, L, seed=seed, walker=w, **kw), spins[w])
        ow.run(12034)
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
    assert not b.status().any()


@pytest.mark.parametrize("box", [0.0, 4.5], ids=["lj", "wca"])
@pytest.mark.parametrize("kw,lanes,max_N", [
    (dict(energy_bin=0.02, min_allowed=-1.0, max_allowed=1.0), 8, 13),
    (dict(energy_bin=0.5, min_allowed=-4.0, max_allowed=3.0, addremove_probability=0.9), 32, 13),
    (dict(energy_bin=0.5, max_allowed=10.0, target_rate=0.5), 16, 40),     # the add/remove threshold moves
    (dict(energy_bin=2.0, max_allowed=20.0, addremove_probability=0.5, method="wl"), 16, 40),
    (dict(energy_bin=0.25, max_allowed=10.0), 32, 60)])
def test_grand_lean_path(gpu, oracle, kw, lanes, max_N, box):
    W, R, seed, runs = 5, 2.5, 9, (6000, 37, 3000)
    kw = dict(dict(t0=500.0, translation_scale=0.1, addremove_probability=0.2, seed=seed), **kw)
    kw["method"] = gpu.WL if kw.get("method") == "wl" else gpu.SAMC
    geo = dict(box=(box,) * 3) if box else {}
    e_lo, e_hi = (-1.0, 25.0) if box else (-200.0, 25.0)
    b = gpu.GrandBatch(gpu.make_grand_config(W, max_N, **(geo or dict(radius=R)), e_lo=e_lo, e_hi=e_hi,
                                             lanes_per_walker=lanes, **kw))
    moves = sum(runs)
    b.set_trace(moves)
    for k in runs:
        b.run(k)
    for w in range(W):
        gs = b.scalars(w)
        assert gs["status"] == 0
        e1, e2 = b.trace(w, moves)
        ow = oracle.GrandWalker(oracle.make_grand_config(**(geo or dict(radius=R)), max_N=max_N, walker=w, **kw))
        disc, mismatch = ow.run_override(e1, e2)
        assert mismatch == 0 and disc < (5e-6 if box else 1e-5), (w, mismatch, disc, ow.worst())
        gb, ob, os_ = b.bins(w), ow.bins(), ow.scalars()
        for k in ("lnw", "hist", "visited", "round_trips"):
            np.testing.assert_array_equal(gb[k], ob[k], err_msg=f"walker {w} {k}")
        for k in SAME:
            assert gs[k] == os_[k], (w, k, gs[k], os_[k])
        for g, o in zip(b.translation_counts(w), ow.translation_counts()):
            np.testing.assert_array_equal(g, o)
        np.testing.assert_allclose(b.state(w), ow.state(), atol=1e-11)


@pytest.mark.parametrize("n,kw", [
    (13, dict(method="sad", energy_bin=0.002, min_allowed=-38.0, max_allowed=-5.0)),
    (33, dict(method="sad", energy_bin=0.3, max_allowed=50.0)),
    (40, dict(method="samc", energy_bin=0.3, min_allowed=-120.0, max_allowed=2.0)),
    (20, dict(method="samc", energy_bin=5.0, max_allowed=0.0)),
    (13, dict(method="wl", energy_bin=2.0, max_allowed=0.0)),
    (64, dict(method="sad", energy_bin=0.2, max_allowed=0.0))], ids=lambda k: k if isinstance(k, int) else k["method"])
def test_delayed_acceptance_lean_path(gpu, oracle, n, kw):
    """Both stages of delayed-acceptance moves, taken by the oracle from the traced energies
    and surrogate changes."""
    W, seed, R, plain, runs = 5, 8, 1.05 * n ** (1 / 3), 2400, (2500, 37, 1000)
    okw = dict(METHOD_KW[kw["method"]], **{k: v for k, v in kw.items() if k != "method"},
               target_rate=0.5, translation_scale=0.1)
    confs = lj_configs(oracle, n, R, range(60, 60 + W))
    b = gpu.Batch(gpu.make_config(gpu.LJ, W, n, e_lo=-6.0 * n - 6, e_hi=kw["max_allowed"] + 6.0, seed=seed,
                                  lanes_per_walker=32, **okw), [(n, R, (0, 0, 0))] * W)
    b.upload(confs)
    b.initialize()
    E0 = b.energies()
    total = plain + sum(runs)
    b.set_trace(total)
    b.surrogate_init(seed=2, ring_capacity=4096)
    for _ in range(6):
        b.run(plain // 6)
        b.surrogate_collect()
    b.surrogate_train(60, batch=64, lr=2e-3, seed=4)
    for k in runs:
        b.run_da(k, refresh_interval=512)
    out_of_range = b.status() & gpu.ST_BIN_RANGE
    assert not out_of_range.all()
    for w in range(W):
        if out_of_range[w]:
            continue  # the reference would have grown its bins
        e1, e2 = b.trace(w, total)
        ds = b.trace_ds(w, total)
        ow = oracle.Walker(oracle.make_config(oracle.LJ, n, radius=R, seed=seed, walker=w, e0=float(E0[w]), **okw),
                           confs[w])
        d1, m1 = ow.run_override(e1[:plain], e2[:plain])
        d2, m2 = ow.run_override_da(e1[plain:], e2[plain:], ds[plain:])
        assert m1 == 0 and m2 == 0 and max(d1, d2) < REPLAY_REL, (w, m1, m2, d1, d2)
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_allclose(b.state(w), ow.state(), atol=1e-11)


@pytest.mark.parametrize("system,lanes", [("ising", 1), ("lj", 8), ("lj", 2), ("wca", 8), ("grand_lj", 8), ("grand_wca", 8)])
def test_few_walkers_run_as_in_a_large_batch(gpu, oracle, system, lanes):
    """A small batch has few walkers per warp, the rest of it repeating their work; a large one
    fills its warps.  A walker's chain is the same."""
    few, runs = 11, (700, 33)
    many = 20000 if lanes == 1 else 11000 if lanes == 2 else 3000

    def batch(W):
        if system.startswith("grand"):
            geo = dict(box=(4.5,) * 3) if system == "grand_wca" else dict(radius=2.5)
            return gpu.GrandBatch(gpu.make_grand_config(W, 20, t0=500.0, energy_bin=0.5, max_allowed=10.0, e_lo=-90.0,
                                                        e_hi=12.0, translation_scale=0.1, addremove_probability=0.2,
                                                        seed=4, lanes_per_walker=lanes, **geo))
        if system == "ising":
            cfg = gpu.make_config(gpu.ISING, W, 8, e_lo=-140.0, e_hi=140.0, seed=4, lanes_per_walker=1,
                                  **METHOD_KW["sad"], energy_bin=4.0)
            geo, confs = (8, 0.0, (0, 0, 0)), [ising_spins(8, w % few) for w in range(W)]
        else:
            n, kind = (13, gpu.LJ) if system == "lj" else (24, gpu.WCA)
            kw = dict(METHOD_KW["sad"], energy_bin=0.5, target_rate=0.5, translation_scale=0.1)
            cfg = gpu.make_config(kind, W, n, e_lo=-60.0 if kind == gpu.LJ else -1.0, e_hi=1.0 if kind == gpu.LJ else 400.0,
                                  max_allowed=0.0 if kind == gpu.LJ else 390.0, seed=4, lanes_per_walker=lanes, **kw)
            if kind == gpu.LJ:
                geo, pool = (n, 2.2, (0, 0, 0)), lj_configs(oracle, n, 2.2, range(40, 40 + few))
            else:
                geo = (n, 0.0, (4.0, 4.0, 4.0))
                pool = [np.random.default_rng(w).permutation(np.stack(np.meshgrid(*[np.arange(3) * 1.3] * 3), -1)
                                                             .reshape(-1, 3))[:n] for w in range(few)]
            confs = [pool[w % few] for w in range(W)]
        b = gpu.Batch(cfg, [geo] * W)
        b.upload(confs)
        b.initialize()
        return b

    a, b = batch(few), batch(many)
    for k in runs:
        a.run(k)
        b.run(k)
    for w in range(few):
        x, y = a.bins(w), b.bins(w)
        for k in x:
            np.testing.assert_array_equal(x[k], y[k], err_msg=f"walker {w} {k}")
        assert a.scalars(w) == b.scalars(w), w
        np.testing.assert_array_equal(a.state(w), b.state(w))
