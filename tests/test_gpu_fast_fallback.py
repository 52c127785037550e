"""Ticks whose particles leave the fast sums' tables, against the FP64 oracle.

A state that fits the tables at the first Stein iterations and overflows them
later: all particles at one point, little state noise and a bandwidth to
match, and SVLD heat that spreads the particles over many panels within the
tick, so that the sweeps over all pairs take over what is left of it.  One
with so many panels that the first iteration does not fit.  Every case checks
on the oracle's own particles when the tables overflow.  Batches run on CTAs of
512 threads and, with a large tile forced on an extra filter, of 256.

Tolerance as in test_gpu_fast_sums: 1e-4 relative (floor 1; KSD 1e-3), or four
times what the oracle's FP32 mirror deviates on the same state and on that state
moved by two FP32 ulps.
"""
import concurrent.futures as cf
import os

import numpy as np
import pytest

import tape
import test_gpu_fast_sums as fast
from test_gpu_batch_parity import _twin
from test_oracle import TOL, rel_err

pytestmark = pytest.mark.gpu

BINS, ZERO, WIDTH, POINTS, FINE = 1024, 512, 0.09375, 12, 8   # csrc/svpf_fast.cuh
MAX_PANELS, MAX_POINTS, MAX_POINTS_2F = 42, 512, 1120
NUDGES = (0.0, 2.0 ** -22, -(2.0 ** -22))


def _overflows(x, two=False):
    """Whether coordinates x (bandwidths) need more panels or points than there is room for."""
    b = np.floor(np.clip(np.asarray(x) / WIDTH, -ZERO, BINS - ZERO - 0.5)).astype(int) + ZERO
    count = np.bincount(b // FINE, minlength=BINS // FINE)
    inter = count > POINTS
    inter[[0, -1]] = False
    points = POINTS * inter.sum() + count[~inter].sum()
    return points > MAX_POINTS_2F if two else inter.sum() > MAX_PANELS or points > MAX_POINTS


def _mirrors(oracle_mod, src, F, cfgs, params):
    out = []
    for nudge in NUDGES:
        m = [_twin(oracle_mod, src, f, cfgs[f], params[f], 1) for f in range(F)]
        for o in m:
            o.h = o.h * (1.0 + nudge)
        out.append(m)
    return out


def _compare(got, twin, mirrors, out, want, around, tag):
    dev = max(rel_err(m.h, twin.h) for m in mirrors)
    assert rel_err(got, twin.h) < max(TOL, 4 * dev), (tag, rel_err(got, twin.h), dev)
    for name, value in out.items():
        w = getattr(want, name)
        base = 1e-3 if name == "ksd" else TOL
        dev = max(abs(getattr(a, name) - w) for a in around) / max(1.0, abs(w))
        assert abs(value - w) < max(base, 4 * dev) * max(1.0, abs(w)), (tag, name, value, w, dev)


def _tick(pkg, oracle_mod, ns, cfgs, params, made, y, yp, slots, narrow):
    """One tick of a batch and of its twins; made(f) -> (ctl changes, h, v)."""
    F = len(ns)
    b = pkg.Batch(list(ns) + [300], list(cfgs) + [cfgs[0]], [pkg.Params(*p) for p in list(params) + [params[0]]])
    b.initialize(seed=3)
    for f in range(F):
        ctl = b.get_state(f)[0]
        changes, h, v = made(f)
        for k, x in changes.items():
            setattr(ctl, k, x)
        b.set_state(f, ctl, h, (h - 0.1).astype(np.float32), v, np.zeros(ns[f], np.float32))
    if narrow:
        b.set_tile(F, 4, 1)   # no one-row tile: the launch runs on CTAs of 256 threads
    nrm, uni = tape.tape(5, 0, max(max(ns), 300), slots, 2)
    b.set_noise_tape(nrm, uni)
    twins = [_twin(oracle_mod, b, f, cfgs[f], params[f]) for f in range(F)]
    mirrors = _mirrors(oracle_mod, b, F, cfgs, params)
    ll, vol, hm = b.step(np.append(y, np.float32(0.3)), np.append(yp, np.float32(0.3)))
    ctl = b.ctl()
    with cf.ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as pool:
        def step(m):
            return list(pool.map(lambda f: m[f].step(y[f], yp[f], nrm[:, :ns[f]], uni[:, :ns[f]]), range(F)))
        want, around = step(twins), [step(m) for m in mirrors]
    for f in range(F):
        out = {"loglik": ll[f], "vol": vol[f], "h_mean": hm[f]}
        if not cfgs[f].use_two_factor:
            out["ksd"] = ctl[f].ksd_last
            assert ctl[f].stein_steps_used == want[f].steps_used, f
        assert ctl[f].status == 0, f
        _compare(b.get_particles(f), twins[f], [m[f] for m in mirrors], out, want[f], [a[f] for a in around],
                 (f, ns[f]))
    b.close()


CTL = dict(timestep=12, ksd_prev=0.6, ksd_last=0.6, vol_prev=0.6, guide_initialized=1, h_mean_prev=-1.0,
           return_ema=0.5, return_var=0.3)
BURST = (0.95, 0.02, -1.0, -0.2)      # particles at one point, hot
TAILS = (0.95, 0.3, -1.0, -0.2)       # a seventh of the particles far out


def _single_state(params, n, rng):
    if params is BURST:
        h = np.full(n, -1.0)
    else:
        h = -1.0 + 0.3 * rng.standard_normal(n)
        h[: n // 7] = rng.uniform(-6.0, 4.0, n // 7)
    v = rng.uniform(0.05, 0.5, n).astype(np.float32)
    return dict(CTL, bw_sq=1e-6 if params is BURST else 1e-4), h.astype(np.float32), v


def _config(pkg, newton):
    cfg = pkg.production_config(8.0, 5)
    cfg.update(use_newton=newton, use_full_newton=newton, stein_min_steps=4, stein_max_steps=4, use_svld=1,
               temperature=0.45)
    return cfg


def _overflow_at(oracle_mod, cfg, params, n, state):
    """The Stein iteration at which the oracle's particles overflow the tables."""
    nrm, uni = tape.tape(5, 0, n, 16, 2)
    for steps in range(4):
        c = oracle_mod.config_from_dict(cfg.to_dict())
        c.stein_min_steps = c.stein_max_steps = steps
        o = oracle_mod.OracleFilter(n, c, oracle_mod.OracleParams(*params), 0)
        for k, x in state[0].items():
            setattr(o.ctl, k, x)
        o.h, o.h_prev = state[1].astype(np.float64), (state[1] - 0.1).astype(np.float64)
        o.v, o.log_w = state[2].astype(np.float64), np.zeros(n)
        o.step(0.4, 0.3, nrm, uni)
        if steps == 0:
            centre = o.h.mean()
        if _overflows((o.h - centre) / o.ctl.bw):
            return steps
    return None


@pytest.mark.parametrize("narrow", [0, 1])
@pytest.mark.parametrize("newton", [1, 0])
def test_batch_ticks_that_leave_the_tables(pkg, oracle_mod, newton, narrow):
    cfg = _config(pkg, newton)
    cases = [(600, BURST), (1025, BURST), (2049, BURST), (4096, BURST), (8192, TAILS)]
    made, when = [], []
    for n, params in cases:
        made.append(_single_state(params, n, np.random.default_rng(n)))
        when.append(_overflow_at(oracle_mod, cfg, params, n, made[-1]))
    assert None not in when and 0 in when and set(when) & {1, 2, 3}, when
    F = len(cases)
    _tick(pkg, oracle_mod, [n for n, _ in cases], [cfg] * F, [p for _, p in cases], lambda f: made[f],
          np.full(F, 0.4, np.float32), np.full(F, 0.3, np.float32), 16, narrow)


@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("n", [2048, 3001, 4096])
def test_single_ticks_that_leave_the_tables(pkg, oracle_mod, n, newton):
    cfg = _config(pkg, newton)
    state = _single_state(BURST, n, np.random.default_rng(n))
    assert _overflow_at(oracle_mod, cfg, BURST, n, state) in (1, 2, 3)
    f = pkg.SVPF(n, 5, 8.0)
    f.configure(**cfg.to_dict())
    f.initialize(*BURST, seed=3)
    ctl = f.get_state()[0]
    for k, x in state[0].items():
        setattr(ctl, k, x)
    f.set_state(ctl, state[1], (state[1] - 0.1).astype(np.float32), state[2], np.zeros(n, np.float32))
    nrm, uni = tape.tape(5, 0, n, 16, 2)
    f.set_noise_tape(nrm, uni)
    twin = _twin(oracle_mod, fast._One(f), 0, cfg, BURST)
    mirrors = [m[0] for m in _mirrors(oracle_mod, fast._One(f), 1, [cfg], [BURST])]
    rc, out = f.step_raw(0.4, 0.3)
    with cf.ThreadPoolExecutor(max_workers=4) as pool:
        want, *around = pool.map(lambda o: o.step(0.4, 0.3, nrm, uni), [twin] + mirrors)
    ctl, got = f.get_state()[:2]
    assert rc == 0 and ctl.status == 0 and ctl.stein_steps_used == want.steps_used
    _compare(got, twin, mirrors, {"loglik": out.loglik, "vol": out.vol, "h_mean": out.h_mean, "ksd": ctl.ksd_last},
             want, around, n)
    f.close()


@pytest.mark.parametrize("narrow", [0, 1])
def test_two_factor_steps_that_leave_the_tables(pkg, oracle_mod, narrow):
    ns = [2048, 3000, 4096]
    cfg = pkg.default_config(2, 6.0)
    cfg.update(use_two_factor=1, rho_fast=0.80, sigma_fast=0.02, rho_slow=0.97, sigma_slow=0.02, bw_floor_fast=0.01,
               bw_floor_slow=0.01, use_svld=1, use_annealing=1, n_anneal_steps=3, temperature=0.45, use_mim=0,
               use_guide=1, guide_strength=0.12, use_exact_gradient=1)
    params = (0.95, 0.1, -3.0, 0.0)
    made = []
    for n in ns:
        rng = np.random.default_rng(n)
        made.append(({}, np.full(2 * n, 0.1, np.float32), rng.uniform(0.05, 0.5, 2 * n).astype(np.float32)))
    nrm, uni = tape.tape(5, 0, max(ns), 24, 2)
    for n, (_, h, v) in zip(ns, made):
        o = oracle_mod.OracleFilter(n, oracle_mod.config_from_dict(cfg.to_dict()), oracle_mod.OracleParams(*params), 0)
        o.h, o.h_prev, o.v, o.log_w = h.astype(float), (h - 0.1).astype(float), v.astype(float), np.zeros(n)
        o.step(0.3, 0.0, nrm[:, :n], uni[:, :n])
        noise = 0.02 * nrm[0, :n]   # the predicted fast factor, but for a shift
        bw = max(1.06 * noise.std() * n ** -0.2, 0.01)
        assert not _overflows((noise - noise.mean()) / bw, True)
        assert _overflows((o.h[:n] - o.h[:n].mean()) / bw, True), n
    _tick(pkg, oracle_mod, ns, [cfg] * 3, [params] * 3, lambda f: made[f], np.full(3, 0.3, np.float32),
          np.zeros(3, np.float32), 24, narrow)


@pytest.mark.parametrize("newton", [1, 0])
@pytest.mark.parametrize("sigma", [0.05, 0.3])
def test_narrow_ctas_match_oracle(pkg, oracle_mod, newton, sigma):
    """The states of test_gpu_fast_sums on CTAs of 256 threads (there: 512)."""
    ns = [n for n in (257, 512, 1025, 2049) for _ in fast.STATES]
    kinds = fast.STATES * 4
    F = len(ns)
    cfg = pkg.production_config(8.0, 5)
    cfg.update(use_newton=newton, use_full_newton=newton, stein_min_steps=4, stein_max_steps=5)
    rng = np.random.default_rng(17)
    made = []
    for f in range(F):
        h = fast._state(kinds[f], ns[f], rng, -1.0)
        made.append((dict(CTL, bw_sq=0.04), h, rng.uniform(0.05, 0.5, ns[f]).astype(np.float32)))
    y = np.array([25.0 if k == "shock" else 0.4 for k in kinds], np.float32)
    _tick(pkg, oracle_mod, ns, [cfg] * F, [(0.95, sigma, -1.0, -0.2)] * F, lambda f: made[f], y,
          np.full(F, 0.3, np.float32), 16, 1)
