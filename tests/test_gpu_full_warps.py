"""Ising batches whose warps are full: the lean path is taken on trial, and a walker's chain is the
same whichever path its moves take.  And the run-time fall-back of the lean path where ln w has
grown past what its binary32 views resolve."""
import numpy as np
import pytest

from helpers import METHOD_KW, assert_bins_equal, assert_scalars_equal, ising_spins

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,L,energy_bin", [("sad", 8, 1.0), ("sad", 9, 3.0), ("samc", 8, 4.0), ("wl", 8, 8.0),
                                                 ("inv_t_wl", 8, 8.0), ("canonical", 8, 4.0)])
def test_full_warps_bit_exact(gpu, oracle, method, L, energy_bin):
    """Fresh walkers, so that the first trials fail and later ones hold; launches that end inside a
    block of 32 moves."""
    W, seed, runs = 20000, 23, (1000, 45, 6000)
    kw = dict(METHOD_KW[method], energy_bin=energy_bin)
    b = gpu.Batch(gpu.make_config(gpu.ISING, W, L, e_lo=-2.0 * L * L - 20, e_hi=2.0 * L * L + 20, seed=seed,
                                  lanes_per_walker=1, **kw), [(L, 0.0, (0, 0, 0))] * W)
    spins = np.where(np.random.default_rng(3).random((W, L * L)) < 0.5, -1.0, 1.0)
    b.upload(list(spins))
    b.initialize()
    for k in runs:
        b.run(k)
    for w in (0, 31, 32, 9999, 19968, 19999):
        ow = oracle.Walker(oracle.make_config(oracle.ISING, L, seed=seed, walker=w, **kw), spins[w])
        ow.run(sum(runs))
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
    assert not b.status().any()


@pytest.mark.parametrize("W", [1, 3])
def test_large_weights(gpu, oracle, W):
    """SAMC with gamma 1 throughout: the few bins of a 2 x 2 lattice pass ln w = 3.3e5, above which
    a binary32 difference of weights no longer decides."""
    L, seed, moves = 2, 29, 1300000
    kw = dict(method=1, t0=1e9, energy_bin=1.0)
    b = gpu.Batch(gpu.make_config(gpu.ISING, W, L, e_lo=-20.0, e_hi=20.0, seed=seed, **kw), [(L, 0.0, (0, 0, 0))] * W)
    spins = [ising_spins(L, 40 + w) for w in range(W)]
    b.upload(spins)
    b.initialize()
    b.run(moves)
    for w in range(W):
        ow = oracle.Walker(oracle.make_config(oracle.ISING, L, seed=seed, walker=w, **kw), spins[w])
        ow.run(moves)
        assert ow.scalars()["max_S"] > 3.4e5
        assert_bins_equal(b.bins(w), ow.bins(), label=f"walker {w}")
        assert_scalars_equal(b.scalars(w), ow.scalars(), label=f"walker {w}")
        np.testing.assert_array_equal(b.state(w), ow.state())
