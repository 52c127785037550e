"""A filter's bits do not depend on the CTA width its launch runs with.

A launch whose largest ticks make it long runs on CTAs of 512 threads instead
of 256, which follows from all its filters.  The same filter must come out of
both with the same particles, moments, control record and outputs, bit for
bit: every sum over particles runs in one order.  A large tile forced on one
filter keeps a batch's launch on CTAs of 256 threads; in the request loop the
number of requests of a round decides.
"""
import numpy as np
import pytest

import cases
from test_gpu_fast_sums import STATES, _state

pytestmark = pytest.mark.gpu


def _made(b, f, n, kind, rng, centre, two):
    ctl = b.get_state(f)[0]
    if not two:
        ctl.timestep, ctl.ksd_prev, ctl.ksd_last, ctl.vol_prev = 12, 0.6, 0.6, 0.6
        ctl.guide_initialized, ctl.h_mean_prev, ctl.bw_sq = 1, -1.0, 0.04
        ctl.return_ema, ctl.return_var = 0.5, 0.3
    h = np.concatenate([_state(kind, n, rng, c) for c in centre])
    v = rng.uniform(0.05, 0.5, len(h)).astype(np.float32)
    b.set_state(f, ctl, h, (h - 0.1).astype(np.float32), v, np.zeros(n, np.float32))


def _run(pkg, ns, kinds, cfg, param, two, narrow, ticks=4):
    b = pkg.Batch(ns, [cfg] * len(ns), [pkg.Params(*param)] * len(ns))
    b.initialize(seed=11)
    rng = np.random.default_rng(29)
    for f, kind in enumerate(kinds):
        _made(b, f, ns[f], kind, rng, (0.0, 0.2) if two else (-1.0,), two)
    if narrow:
        b.set_tile(len(ns) - 1, 4, 1)   # no one-row tile: the launch runs on CTAs of 256 threads
    outs, y, yp = [], None, np.zeros(len(ns), np.float32)
    for t in range(ticks):
        y = (0.3 + 0.04 * np.arange(len(ns)) % 0.7 + 0.2 * t).astype(np.float32)
        outs.append(b.step(y, yp))
        yp = y
    state = [b.get_state(f) for f in range(len(ns))]
    b.close()
    return outs, state


def _same(a, b, tag):
    for x, y in zip(a, b):
        x, y = (bytes(v) if not isinstance(v, np.ndarray) else v.tobytes() for v in (x, y))
        assert x == y, tag


@pytest.mark.parametrize("kind", STATES)
@pytest.mark.parametrize("newton", [1, 0])
def test_batch_bits_do_not_depend_on_the_width(pkg, newton, kind):
    ns = [100, 200, 256, 257, 300, 511, 512, 513, 777, 1025, 2049, 4096, 300]
    cfg = pkg.production_config(8.0, 5)
    cfg.update(use_newton=newton, use_full_newton=newton, stein_min_steps=3, stein_max_steps=6)
    for sigma in (0.05, 0.3):
        (o1, s1), (o2, s2) = (_run(pkg, ns, [kind] * (len(ns) - 1), cfg, (0.95, sigma, -1.0, -0.2), False, nar)
                              for nar in (False, True))
        for t in range(len(o1)):
            for a, b in zip(o1[t], o2[t]):
                assert a[:-1].tobytes() == b[:-1].tobytes(), (t, sigma, ns, a - b)
        for f in range(len(ns) - 1):
            _same(s1[f], s2[f], (ns[f], sigma))


@pytest.mark.parametrize("kind", ["cloud", "point", "outliers", "clamped", "spread"])
def test_two_factor_bits_do_not_depend_on_the_width(pkg, kind):
    ns = [64, 200, 256, 257, 300, 513, 777, 1025, 2048, 300]
    cfg = pkg.default_config(2, 6.0)
    cfg.update(**dict(cases.TWO_FACTOR_TEST, n_anneal_steps=3, nu=6.0, rho_fast=0.80, sigma_fast=0.30, rho_slow=0.97,
                      sigma_slow=0.10))
    (o1, s1), (o2, s2) = (_run(pkg, ns, [kind] * (len(ns) - 1), cfg, (0.95, 0.1, -3.0, 0.0), True, nar)
                          for nar in (False, True))
    for t in range(len(o1)):
        for a, b in zip(o1[t], o2[t]):
            assert a[:-1].tobytes() == b[:-1].tobytes(), (t, a - b)
    for f in range(len(ns) - 1):
        _same(s1[f], s2[f], ns[f])


def test_an_instrument_does_not_depend_on_its_round(pkg):
    """All instruments in one round (enough ticks for CTAs of 256 threads), in
    rounds of 16, and from device buffers."""
    torch = pytest.importorskip("torch")
    F1 = F2 = 260
    one = pkg.production_config(8.0, 5)
    one.update(stein_min_steps=2, stein_max_steps=4)
    two = pkg.default_config(2, 6.0)
    two.update(**dict(cases.TWO_FACTOR_TEST, n_anneal_steps=2, nu=6.0, rho_fast=0.80, sigma_fast=0.30, rho_slow=0.995,
                      sigma_slow=0.05))
    ns = [(300, 301, 290)[f % 3] for f in range(F1 + F2)]
    loops = []
    for _ in range(3):
        s = pkg.Stream(F1 + F2, 64 << 20, 512, seed=7)
        for f in range(F1 + F2):
            prm = pkg.Params(0.97, 0.15, -1.0, -0.1) if f < F1 else pkg.Params(0.995, 0.05, -3.5, 0.0)
            assert s.admit(ns[f], one if f < F1 else two, prm, seed=7) == f
        loops.append(s)
    whole, parts, device = loops
    F = F1 + F2
    rng = np.random.default_rng(3)
    ids = np.arange(F, dtype=np.int32)
    for t in range(4):
        y = (0.5 * rng.standard_normal(F)).astype(np.float32)
        whole.process(ids, y)
        for k in range(0, F, 16):
            parts.process(ids[k:k + 16], y[k:k + 16])
        d_slots, d_y = torch.tensor(ids, device="cuda"), torch.tensor(y, device="cuda")
        d_out = torch.zeros((F, 8), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        device.process_device(F1, F2, d_slots.data_ptr(), d_y.data_ptr(), d_out.data_ptr())
        torch.cuda.synchronize()
    for f in range(F):
        want = whole.particles(f).tobytes(), bytes(whole.ctl(f))
        for s in (parts, device):
            assert (s.particles(f).tobytes(), bytes(s.ctl(f))) == want, f
    for s in loops:
        s.close()
