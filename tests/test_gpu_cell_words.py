"""The periodic-cell moves where a bucket's word holds fewer atoms than the bucket (more than
four in a subcell), where a grid has the fewest subcells (three per axis, every query wraps)
and for every number of lanes per walker, against the FP64 oracle; and a checkpoint resumed
into a run (the words are rebuilt from the saved lists)."""
import numpy as np
import pytest

from helpers import assert_bins_equal, assert_scalars_equal

pytestmark = pytest.mark.gpu


def jittered(m, n, edge, seed, jitter):
    rng = np.random.default_rng(seed)
    g = np.indices((m, m, m)).reshape(3, -1).T.astype(float)
    g = g[rng.permutation(len(g))[:n]]
    return np.mod((g + 0.5 + rng.uniform(-jitter, jitter, g.shape)) * (edge / m), edge)


@pytest.mark.parametrize("lpw", [4, 8, 16, 32])
def test_full_buckets_square_well_bit_exact(gpu, oracle, lpw, tmp_path):
    W, well, seed, runs = 5, 1.9, 5, (1500, 45, 2000)
    specs = [(125, 5.76), (120, 5.8), (90, 5.9), (125, 7.7), (60, 5.75)]  # 3 or 4 subcells per axis
    confs = [jittered(5, n, edge, 60 + w, 0.01) for w, (n, edge) in enumerate(specs)]
    kw = dict(method=2, well_width=well, translation_scale=0.12, seed=seed)
    b = gpu.Batch(gpu.make_config(gpu.SW, W, 125, e_lo=-2600.0, e_hi=2.0, lanes_per_walker=lpw, **kw),
                  [(n, 0.0, (edge,) * 3) for n, edge in specs])
    b.upload(confs)
    b.initialize()
    b.run(runs[0])
    path = str(tmp_path / "cells.ck")
    b.checkpoint(path)
    b = gpu.Batch.resume(path)
    for k in runs[1:]:
        b.run(k)
    for w, (n, edge) in enumerate(specs):
        ow = oracle.Walker(oracle.make_config(oracle.SW, n, box=(edge,) * 3, walker=w, **kw), confs[w])
        ow.run(sum(runs))
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
    np.testing.assert_array_equal(b.energies(), b.compute_energies())
    assert not b.status().any()


@pytest.mark.parametrize("lpw", [4, 8, 16, 32])
@pytest.mark.parametrize("method", ["sad", "wl"])
def test_full_buckets_wca_trace_replay(gpu, oracle, lpw, method):
    W, seed, w_bin, runs = 3, 6, 1.0, (700, 33, 500)
    specs = [(64, 4.42), (75, 4.45), (60, 4.4)]  # three subcells of about 1.5 per axis
    confs = [jittered(5, n, edge, 80 + w, 0.05) for w, (n, edge) in enumerate(specs)]
    kw = dict(method={"sad": 0, "wl": 2}[method], min_T=0.5, energy_bin=w_bin, max_allowed=1500.0,
              translation_scale=0.1, seed=seed)
    b = gpu.Batch(gpu.make_config(gpu.WCA, W, 75, e_lo=-2 * w_bin, e_hi=1700.0, lanes_per_walker=lpw,
                                  resum_interval=400, **kw), [(n, 0.0, (edge,) * 3) for n, edge in specs])
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
