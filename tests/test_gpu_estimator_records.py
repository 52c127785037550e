"""The estimator's two ways to the backward give the same bits.

An engine whose T_max makes its run records larger than 4 GiB takes
checkpoints; one made for the run's own length takes the records.  Enough paths
to fill the GPU several times, and particle counts around the blocks of 64 that
the records are padded to.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps", [(2, 2), (62, 0), (64, 2), (66, 1), (100, 2), (128, 3), (130, 2), (256, 2), (258, 2)])
def test_records_and_checkpoints_agree(pkg, n, steps):
    F, T = 592, 40
    rng = np.random.default_rng(n)
    theta = np.stack([rng.uniform(-2.0, 0.0, F), rng.uniform(0.8, 0.97, F), rng.uniform(0.1, 0.4, F),
                      rng.uniform(4.0, 20.0, F)], 1).astype(np.float32)
    y = (0.5 * rng.standard_normal((F, T))).astype(np.float32)
    floats = (4 + max(steps, 1)) * ((n + 63) // 64 * 64) + 4
    too_long = (4 << 30) // (4 * F * floats) + 1
    got = []
    for T_max in (T, too_long):
        e = pkg.Estimator(F, n, n_stein_steps=steps, T_max=T_max, checkpoint_every=16, truncate_every=15)
        ll, vol, total = e.forward(theta, y, seed=5)
        got.append((ll, vol, total, e.backward()))
        e.close()
    for a, b in zip(*got):
        assert a.tobytes() == b.tobytes(), np.abs(a - b).max()
