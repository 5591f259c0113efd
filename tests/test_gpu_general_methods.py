"""The methods without a lean path (canonical, 1/t-WL), which have kernels of their own, against
the FP64 oracle; 1/t-WL walkers switch to SAMC in the middle of a run."""
import numpy as np
import pytest

from helpers import METHOD_KW, assert_bins_equal, assert_scalars_equal, ising_spins
from test_gpu_cell_words import jittered

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W", [1, 5])
@pytest.mark.parametrize("method", ["inv_t_wl", "canonical"])
def test_ising_switches_to_samc(gpu, oracle, method, W):
    L, seed, runs = 4, 21, (20011, 40000)
    kw = dict(METHOD_KW[method], energy_bin=8.0)
    b = gpu.Batch(gpu.make_config(gpu.ISING, W, L, e_lo=-52.0, e_hi=52.0, seed=seed, **kw), [(L, 0.0, (0, 0, 0))] * W)
    spins = [ising_spins(L, 900 + w) for w in range(W)]
    b.upload(spins)
    b.initialize()
    for k in runs:
        b.run(k)
    for w in range(W):
        ow = oracle.Walker(oracle.make_config(oracle.ISING, L, seed=seed, walker=w, **kw), spins[w])
        ow.run(sum(runs))
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
        if method == "inv_t_wl":
            assert ow.scalars()["method_kind"] == gpu.SAMC
    assert not b.status().any()


@pytest.mark.parametrize("lpw", [4, 8, 16, 32])
@pytest.mark.parametrize("method", ["inv_t_wl", "canonical"])
def test_square_well_bit_exact(gpu, oracle, method, lpw):
    W, seed, runs = 3, 5, (1500, 45)
    specs = [(125, 5.76), (120, 5.8), (60, 5.75)]
    confs = [jittered(5, n, edge, 60 + w, 0.01) for w, (n, edge) in enumerate(specs)]
    kw = dict(METHOD_KW[method], well_width=1.9, translation_scale=0.12, seed=seed)
    b = gpu.Batch(gpu.make_config(gpu.SW, W, 125, e_lo=-2600.0, e_hi=2.0, lanes_per_walker=lpw, **kw),
                  [(n, 0.0, (edge,) * 3) for n, edge in specs])
    b.upload(confs)
    b.initialize()
    for k in runs:
        b.run(k)
    for w, (n, edge) in enumerate(specs):
        ow = oracle.Walker(oracle.make_config(oracle.SW, n, box=(edge,) * 3, walker=w, **kw), confs[w])
        ow.run(sum(runs))
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
    assert not b.status().any()


@pytest.mark.parametrize("lpw", [8, 32])
@pytest.mark.parametrize("method", ["inv_t_wl", "canonical"])
def test_wca_trace_replay(gpu, oracle, method, lpw):
    W, seed, runs = 3, 6, (700, 33)
    specs = [(64, 4.42), (75, 4.45), (60, 4.4)]
    confs = [jittered(5, n, edge, 80 + w, 0.05) for w, (n, edge) in enumerate(specs)]
    kw = dict(METHOD_KW[method], energy_bin=1.0, max_allowed=1500.0, translation_scale=0.1, seed=seed)
    b = gpu.Batch(gpu.make_config(gpu.WCA, W, 75, e_lo=-2.0, e_hi=1700.0, lanes_per_walker=lpw, resum_interval=400,
                                  **kw), [(n, 0.0, (edge,) * 3) for n, edge in specs])
    b.upload(confs)
    b.initialize()
    E0 = b.energies()
    b.set_trace(sum(runs))
    for k in runs:
        b.run(k)
    for w, (n, edge) in enumerate(specs):
        e1, e2 = b.trace(w, sum(runs))
        ow = oracle.Walker(oracle.make_config(oracle.WCA, n, box=(edge,) * 3, walker=w, e0=float(E0[w]), **kw),
                           confs[w])
        disc, mismatch = ow.run_override(e1, e2)
        # the bound of test_gpu_cells.py on the double-single pair differences
        assert mismatch == 0 and disc < 5e-6, (w, mismatch, disc)
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_allclose(b.state(w), ow.state(), atol=1e-12)
    assert not b.status().any()
