"""The constants of the panel interpolation (csrc/svpf_fast.cuh), on the CPU.

kBasis must be the inverse of the Chebyshev matrix at the points kNode, which it
is computed from here again in rational arithmetic, and the interpolation of
each pair sum's kernel from kNode must leave the error that the source states.
"""
import os
import re
from fractions import Fraction

import numpy as np

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "newton-stein-variational-particle-filter_b200", "csrc", "svpf_fast.cuh")
TEXT = open(SRC).read()
P = 12
WIDTH = 0.75   # panel width in bandwidths


def _array(name):
    body = re.search(r"float %s\[[^\]]*\] = \{(.*?)\};" % name, TEXT, re.S).group(1)
    return [x.strip().rstrip("f") for x in body.split(",")]


def _inverse(m):
    n = len(m)
    a = [row[:] + [Fraction(int(i == j)) for j in range(n)] for i, row in enumerate(m)]
    for c in range(n):
        p = max(range(c, n), key=lambda r: abs(a[r][c]))
        a[c], a[p] = a[p], a[c]
        a[c] = [x / a[c][c] for x in a[c]]
        for r in range(n):
            if r != c and a[r][c] != 0:
                a[r] = [x - a[r][c] * y for x, y in zip(a[r], a[c])]
    return [row[n:] for row in a]


def _cheb(t, one):
    out = [one, t]
    while len(out) < P:
        out.append(2 * t * out[-1] - out[-2])
    return out


NODE = [Fraction(x) for x in _array("kNode")]
BASIS = np.array([float(x) for x in _array("kBasis")]).reshape(P, P)


def test_points_are_multiples_of_2_to_the_minus_14():
    assert all((x * 2 ** 14).denominator == 1 and abs(x) < Fraction(3, 8) for x in NODE)
    assert NODE == [-x for x in reversed(NODE)]


def test_basis_is_the_inverse_of_the_chebyshev_matrix():
    """Written with ten digits: half a unit of the last one is 5e-11 of a value below 0.2."""
    inv = _inverse([_cheb(x / Fraction(3, 8), Fraction(1)) for x in NODE])   # points by degrees -> degrees by points
    want = np.array([[float(x) for x in row] for row in inv])
    assert np.abs(BASIS - want).max() < 6e-11, np.abs(BASIS - want).max()


def test_interpolation_error_of_the_pair_kernels():
    """Largest error of an interpolated kernel value over sources and panel
    positions, relative to the kernel's largest value."""
    inv = np.array([[float(x) for x in row] for row in
                    _inverse([_cheb(x / Fraction(3, 8), Fraction(1)) for x in NODE])])
    node = np.array([float(x) for x in NODE])
    x = np.linspace(-WIDTH / 2, WIDTH / 2, 401)
    T = np.stack(_cheb(x / (WIDTH / 2), np.ones_like(x)), 1)
    src = np.linspace(-6.0, 6.0, 2401)[:, None]

    def K(u):
        return 1.0 / (1.0 + u * u)

    kernels = {"K": (K, 2.6e-9), "u K^2": (lambda u: u * K(u) ** 2, 1.5e-8),
               "K (3 - 4K)": (lambda u: K(u) * (3 - 4 * K(u)), 6.1e-8),
               "K^2 (3 - 4K)": (lambda u: K(u) ** 2 * (3 - 4 * K(u)), 2.1e-7)}
    for name, (f, bound) in kernels.items():
        err = np.abs(f(node - src) @ inv.T @ T.T - f(x - src)).max()
        print(name, err)
        assert err < bound, (name, err)
