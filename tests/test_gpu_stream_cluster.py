"""Two-factor instruments whose fast layout does not fit one CTA run on 4-CTA
clusters in the request loop (6465 to 6784 particles): against the same filter
by itself, which sweeps on a cluster of 16, and beside one that takes the fast
sums on one CTA."""
import numpy as np
import pytest

import cases
from test_oracle import TOL, rel_err

pytestmark = pytest.mark.gpu
SEED = 7


@pytest.mark.parametrize("n", [6465, 6784])
def test_largest_two_factor_instruments(pkg, n):
    cfg = pkg.default_config(4, 6.0)
    cfg.update(**dict(cases.TWO_FACTOR_TEST, n_anneal_steps=2, nu=6.0, rho_fast=0.80, sigma_fast=0.30,
                      rho_slow=0.995, sigma_slow=0.05))
    prm = (0.995, 0.05, -3.5, 0.0)
    s = pkg.Stream(2, 64 << 20, n, seed=SEED)
    assert [s.admit(k, cfg, pkg.Params(*prm), seed=SEED) for k in (n, 2048)] == [0, 1]
    f = pkg.SVPF(n, 4, 6.0)
    f.configure(**cfg.to_dict())
    f.initialize(*prm, seed=SEED)
    b = pkg.Batch([300, 2048], [cfg, cfg], [pkg.Params(*prm)] * 2)
    b.initialize(seed=SEED)
    yp = 0.0
    for y in (0.01, -0.03, 0.02):
        launches = s.kernel_launches
        out = s.process(np.arange(2), np.full(2, y, np.float32))
        assert s.kernel_launches == launches + 2   # the cluster's and the one-CTA kernel
        rc, want = f.step_raw(y, yp)
        ll, _, hm = b.step(np.full(2, y, np.float32), np.full(2, yp, np.float32))
        assert rc == 0
        for got, w_ll, w_hm in ((out[0], want.loglik, want.h_mean), (out[1], ll[1], hm[1])):
            assert abs(got.loglik - w_ll) <= TOL * max(1, abs(w_ll)), (y, got.loglik, w_ll)
            assert abs(got.h_mean - w_hm) <= TOL * max(1, abs(w_hm)), (y, got.h_mean, w_hm)
        yp = y
    assert rel_err(s.particles(0), f.get_state_2f()[0]) < TOL
    assert rel_err(s.particles(1), b.get_particles(1)) < TOL
    for x in (s, f, b):
        x.close()
