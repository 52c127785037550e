"""Host-side choices of the library on a fake CUDA runtime (no GPU needed)."""
from host_fake import on_fake  # noqa: F401


def test_largest_heun_filter_is_accepted(on_fake):  # noqa: F811
    """What a kernel's static variables leave of the 227 KB holds a Heun
    filter of 7076 particles, the largest that its layout allows."""
    on_fake(r"""
cfg = pkg.default_config(2, 8.0)
cfg.update(use_heun=1)
assert created(lambda: pkg.Batch([7076], [cfg], [pkg.Params(0.95, 0.1, -1.0, 0.0)]))
assert not created(lambda: pkg.Batch([7077], [cfg], [pkg.Params(0.95, 0.1, -1.0, 0.0)]))
""")


def test_two_factor_instruments_take_the_fast_sums_in_a_loop_of_any_size(on_fake):  # noqa: F811
    """An instrument of 2048 particles runs on one CTA through the fast sums
    whatever n_max the loop was made for; one whose fast layout does not fit
    takes a cluster.  What a loop refuses stays refused."""
    on_fake(r"""
cfg = pkg.default_config(2, 6.0)
cfg.update(use_two_factor=1, rho_fast=0.8, sigma_fast=0.3, rho_slow=0.97, sigma_slow=0.1)
prm = pkg.Params(0.95, 0.1, -3.0, 0.0)

def kernels(s, slots):
    launches()
    s.process(np.array(slots, np.int32), np.full(len(slots), 0.3, np.float32))
    return [(("cluster" in name), block, smem) for name, _, block, smem in launches() if "batch_tick_2f" in name]

for n_max in (2048, 4096, 5760, 5761, 6000, 6464, 6465, 6784):
    s = pkg.Stream(4, 64 << 20, n_max, seed=1)
    a = s.admit(2048, cfg, prm)
    ran = kernels(s, [a])
    assert len(ran) == 1 and not ran[0][0], (n_max, ran)
    if n_max > 5760:
        b = s.admit(n_max, cfg, prm)
        ran = kernels(s, [a, b])
        assert sorted(k for k, _, _ in ran) == ([False, True] if n_max > 6464 else [False]), (n_max, ran)
        assert s.admit(1023, cfg, prm) < 0
        d = np.zeros(64, np.float32)
        try:
            s.process_device(0, 1, d.ctypes.data, d.ctypes.data, d.ctypes.data)
            raise SystemExit("launched")
        except RuntimeError:
            pass
    s.close()
""")


def test_estimator_leaves_its_records_to_what_else_needs_the_memory(on_fake):  # noqa: F811
    """A record of every tick speeds the backward up; an engine that fits
    without it is created, and takes a noise tape, where the memory for it is
    short, and never takes most of what is free."""
    on_fake(r"""
F, T, n = 256, 100, 64
records = F * T * (6 * 64 + 4) * 4          # 39.7 MB
theta = np.tile(np.array([-1.0, 0.95, 0.2, 8.0], np.float32), (F, 1))
y = np.full((F, T), 0.3, np.float32)

def way(e, tape=None):
    launches()
    e.forward(theta, y, tape=tape)
    e.backward()
    return "records" if len(launches()) == 2 else "checkpoints"

e = pkg.Estimator(F, n, T_max=T)
assert way(e) == "records"
used = fake.fake_memory_used()
e.close()
for spare in (0, 1 << 16, 1 << 20, 4 << 20):            # room for the records, and for part of the rest
    fake.fake_set_memory(records + spare)
    e = pkg.Estimator(F, n, T_max=T)
    assert way(e) == "checkpoints", spare
    e.close()
fake.fake_set_memory(used)                   # no room for a tape of 3.4 MB beside them
e = pkg.Estimator(F, n, T_max=T)
assert way(e) == "records"
assert way(e, np.zeros((F, e.tape_floats(n, T)), np.float32)) == "checkpoints"
e.close()
assert fake.fake_memory_used() == 0
for room, want in ((64 << 30, "records"), (1 << 30, "checkpoints")):   # 159 MB of records
    fake.fake_set_memory(room)
    e = pkg.Estimator(4 * F, n, T_max=T)
    theta, y = np.tile(theta[:1], (4 * F, 1)), np.full((4 * F, T), 0.3, np.float32)
    assert way(e) == want, room
    e.close()
""")
