"""Delayed-acceptance moves from a walker's first move on: the second-stage uniforms are
drawn for every move, not only once the move count has passed a batch."""
import numpy as np
import pytest

from helpers import METHOD_KW, assert_bins_equal, assert_scalars_equal, lj_configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,plain,runs", [(13, 0, (29, 3, 1, 200)), (38, 0, (400,)), (20, 7, (1, 60))])
def test_delayed_acceptance_from_the_first_move(gpu, oracle, n, plain, runs):
    """The oracle replays the traced energies and surrogate changes and takes both stages'
    decisions itself, from its own draws.  The surrogate is an untrained one with a steep last
    layer, whose changes are bins away from the exact ones: the first stage accepts uphill
    moves, and the second rejects some of them."""
    W, seed, R = 96, 31, 1.05 * n ** (1 / 3)
    kw = dict(METHOD_KW["samc"], energy_bin=0.5, max_allowed=0.0, target_rate=0.5, translation_scale=0.1)
    confs = lj_configs(oracle, n, R, range(80, 80 + W))
    b = gpu.Batch(gpu.make_config(gpu.LJ, W, n, e_lo=-6.0 * n - 6, e_hi=6.0, seed=seed, lanes_per_walker=32, **kw),
                  [(n, R, (0, 0, 0))] * W)
    b.upload(confs)
    b.initialize()
    E0 = b.energies()
    total = plain + sum(runs)
    b.set_trace(total)
    b.surrogate_init(seed=2)
    params = b.surrogate_params()
    params[-65:-1] *= 10.0
    b.surrogate_set_params(params)
    if plain:
        b.run(plain)
    for k in runs:
        b.run_da(k)
    assert not b.status().any()
    second_stage_rejected = 0
    for w in range(W):
        e1, e2 = b.trace(w, total)
        ds = b.trace_ds(w, total)
        ow = oracle.Walker(oracle.make_config(oracle.LJ, n, radius=R, seed=seed, walker=w, e0=float(E0[w]), **kw), confs[w])
        d1, m1 = ow.run_override(e1[:plain], e2[:plain])
        d2, m2 = ow.run_override_da(e1[plain:], e2[plain:], ds[plain:])
        assert m1 == 0 and m2 == 0 and max(d1, d2) < 2e-5, (w, m1, m2, d1, d2)
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_allclose(b.state(w), ow.state(), atol=1e-11)
        tried = np.isfinite(e2[plain:-1])
        second_stage_rejected += int((tried & (e1[plain + 1:] == e1[plain:-1])).sum())
    assert second_stage_rejected > W
