"""The warm split's polish accepts a basis only if the one Newton-Schulz step it makes leaves it
orthonormal to the tolerance, in every entry.

Bases Z with a chosen E = Z^T Z - 1 on both sides of the decision; the deviation after the step is
formed from E itself, (1 - E/2)^2 (1 + E) - 1 = -3/4 E^2 + 1/4 E^3, without a difference to lose digits in.
"""
import ctypes

import numpy as np
import pytest

from internal import load, ptr

pytestmark = pytest.mark.gpu


def _decide(E, tol, K):
    k = E.shape[0]
    S = np.full((K, K), 7.0)  # nothing beyond the leading block counts
    S[:k, :k] = np.eye(k) + E
    flags = (ctypes.c_int * 2)()
    assert load().probe_ns_check(ptr(S), K, k, ctypes.c_double(tol), flags) == 0
    return flags[0], flags[1]


def _pattern(kind, k, rng):
    if kind == "random":
        E = rng.standard_normal((k, k))
        E = E + E.T
    elif kind == "uniform":  # every entry as large as the largest
        s = rng.choice([-1.0, 1.0], k)
        E = np.outer(s, s)
    elif kind == "row":
        E = np.zeros((k, k))
        E[k // 2] = E[:, k // 2] = 1.0
    else:
        E = np.diag(rng.standard_normal(k))
    return E / np.abs(E).max()


@pytest.mark.parametrize("kind", ["random", "uniform", "row", "diagonal"])
@pytest.mark.parametrize("k,K", [(1, 1), (31, 40), (64, 64), (256, 256), (300, 333), (512, 512)])
def test_accepted_step_is_within_tolerance(kind, k, K):
    rng = np.random.default_rng(k)
    E = _pattern(kind, k, rng)
    tol = 4e-16 * 2 * k
    E2 = E @ E
    E3 = E2 @ E
    accepted = rejected = 0
    for t in np.sqrt(tol) * np.geomspace(0.3 / k, 2.0, 25):
        done, near = _decide(t * E, tol, K)
        dev = np.abs(-0.75 * t * t * E2 + 0.25 * t ** 3 * E3).max()
        assert not done or t < tol
        if near:
            assert dev < 0.4 * tol * (1.0 + 1e-6)  # the rest of the tolerance is for rounding
            accepted += 1
        else:
            # the bound is attained on the diagonal of E^2, so little that would pass is refused
            assert dev > 0.39 * tol
            rejected += 1
    assert accepted and rejected


def test_orthonormal_and_undefined_blocks():
    E = np.zeros((65, 65))
    assert _decide(E, 1e-14, 70) == (1, 1)
    E[3, 60] = np.nan
    assert _decide(E, 1e-14, 70)[1] == 0
