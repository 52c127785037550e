"""The default cluster of a single filter against the FP64 oracle at the sizes
around which its choice changes (1, 4, 8 and 16 CTAs), three ticks each from a
re-synced state.  Tolerance: 1e-4 relative (floor 1), KSD 1e-3."""
import numpy as np
import pytest

import tape
from test_gpu_parity import CONFIGS, engine_for, oracle_twin
from test_oracle import TOL, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cfg_name", ["production", "vanilla"])
@pytest.mark.parametrize("n", [64, 65, 128, 129, 256, 257, 511])
def test_default_cluster_matches_oracle(pkg, oracle_mod, n, cfg_name):
    params = (0.97, 0.15, -1.0, -0.1)
    f = engine_for(pkg, n, 8, 30.0, {}, params)
    f.configure(**{k: getattr(pkg.default_config(8, 30.0), k) for k, _ in pkg.CONFIG_FIELDS})
    f.configure(**CONFIGS[cfg_name])
    f.set_noise_tape(tape.init_normals(11, n)[None, :], np.ones((1, n), np.float32))
    f.initialize(*params, seed=5)
    _, ys = tape.sv_path(4, -1.0, 0.97, 0.15, seed=n)
    y_prev = 0.0
    for t in range(3):
        o = oracle_twin(oracle_mod, pkg, f, params)
        nrm, uni = tape.tape(99, t, n, 9 + f.config.stein_max_steps, 2)
        f.set_noise_tape(nrm, uni)
        rc, out = f.step_raw(ys[t], y_prev)
        want = o.step(ys[t], y_prev, nrm, uni)
        y_prev = float(ys[t])
        assert rc == 0 and out.steps_used == want.steps_used
        assert rel_err(f.get_particles(), o.h) < TOL, t
        assert abs(out.loglik - want.loglik) < TOL * max(1, abs(want.loglik)), t
        assert abs(out.ksd - want.ksd) < 1e-3 * max(1, abs(want.ksd)), t
    f.close()
