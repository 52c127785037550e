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
