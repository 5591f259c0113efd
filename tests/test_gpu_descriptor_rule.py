"""Predictions on either side of the sizes where the descriptors change kernel: the values do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,configs", [(42, 2559), (42, 2560), (43, 6143), (43, 6144), (51, 6145), (52, 6144)])
def test_descriptor_kernels_agree(gpu, n, configs):
    """A pair's term serves both of its atoms in one kernel and is taken per atom in the other, in
    the same order of a row's sum; batches of 700 configurations take the other one."""
    R = 1.2 * n ** (1 / 3)
    b = gpu.Batch(gpu.make_config(gpu.LJ, 1, n, energy_bin=0.5, max_allowed=0.0, e_lo=-6.0 * n, e_hi=1.0, seed=2),
                  [(n, R, (0, 0, 0))])
    b.surrogate_init(seed=4, ring_capacity=16)
    pos = np.random.default_rng(n).normal(0, R / 2, (configs, n, 3)).astype(np.float32)
    got = b.surrogate_predict(pos)
    small = np.concatenate([b.surrogate_predict(pos[k:k + 700]) for k in range(0, configs, 700)])
    np.testing.assert_array_equal(got, small)
