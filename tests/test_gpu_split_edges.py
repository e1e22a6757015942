"""Edges of the GEMM tiles and of the split kernels, against numpy.

GEMMs: shapes that the tile model sends to each tile and to clustered K splits, with remainders in
every dimension and odd leading dimensions (8-byte copies) on either operand; the error of a dot
product of K terms stays below K eps |a||b|.
Splits: orders around the one-launch Newton-Schulz block (64), the tile of the Cholesky factor (32)
and its cluster sizes (256), real and complex.
"""
import numpy as np
import pytest

import dmrg2

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


def _rnd(rng, shape, cplx):
    x = rng.standard_normal(shape)
    return x + 1j * rng.standard_normal(shape) if cplx else x


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("ta,tb", [("N", "N"), ("N", "T"), ("T", "N"), ("T", "T"), ("C", "T")])
@pytest.mark.parametrize("shape", [(33, 31, 1), (40, 44, 1500), (97, 66, 641), (700, 610, 40), (1281, 130, 33),
                                   (640, 512, 128), (131, 1025, 255)])
def test_gemm_tiles(shape, ta, tb, cplx):
    if ta == "C" and not cplx:
        pytest.skip("conjugation needs complex data")
    M, N, K = shape
    rng = np.random.default_rng(7)
    A = _rnd(rng, (M, K) if ta == "N" else (K, M), cplx)
    B = _rnd(rng, (K, N) if tb == "N" else (N, K), cplx)
    C0 = _rnd(rng, (M, N), cplx)
    opA = A if ta == "N" else (A.T if ta == "T" else A.conj().T)
    opB = B if tb == "N" else B.T
    al, be = (0.7 - 0.2j, -0.5 + 1.1j) if cplx else (0.7, -0.5)
    out = dmrg2.gemm(A, B, ta, tb, alpha=al, beta=be, C=C0)
    bound = (np.abs(opA) @ np.abs(opB)) * abs(al) + np.abs(C0) * abs(be)
    assert np.all(np.abs(out - (al * (opA @ opB) + be * C0)) <= (2 * K + 8) * EPS * bound)


@pytest.mark.parametrize("shape", [(1024, 256, 1280), (684, 187, 1496), (1000, 240, 1200), (700, 250, 1500)])
def test_long_sums_are_split(shape):
    """H_eff's last step sums over D chi values. Against one chain of fused multiply-adds over them (formed
    here, rounded at each addition), slices of at most 384 leave at most sqrt(384 / K) of its error (outputs
    of fewer 64 x 64 tiles than SMs)."""
    M, N, K = shape
    rng = np.random.default_rng(9)
    A, B = rng.standard_normal((M, K)), rng.standard_normal((N, K))
    rows = np.arange(0, M, 37)
    a, b = A[rows].astype(np.longdouble), B.T.astype(np.longdouble)
    exact = a @ b
    chain = np.zeros(exact.shape)
    for k in range(K):
        chain = (chain + a[:, k:k + 1] * b[k]).astype(np.float64)
    err = np.linalg.norm((dmrg2.gemm(A, B, "N", "T")[rows] - exact).astype(np.float64))
    one = np.linalg.norm((chain - exact).astype(np.float64))
    assert err <= 1.15 * np.sqrt(384.0 / K) * one  # (15%: the sum over the slices, and the sample)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 31, 63, 64, 65, 128, 129])
def test_exact_split_orders(n, cplx):
    rng = np.random.default_rng(n)
    U, _ = np.linalg.qr(_rnd(rng, (n, n), cplx))
    V, _ = np.linalg.qr(_rnd(rng, (n, n), cplx))
    s = np.exp(-6.0 * np.arange(n) / n)
    M = (U * s) @ V.conj().T
    k = max(1, n // 2)
    left, S, right, te = dmrg2.truncated_svd(M, k, 0.0, "R")
    # the density matrix squares the spectrum: eps s_0^2 / s_i on a singular value, s_i >= e^-6 s_0
    assert np.abs(S - s).max() < 1e-12
    assert np.abs(left.conj().T @ left - np.eye(k)).max() < 1e-12
    assert np.abs(left @ (left.conj().T @ M) - (U[:, :k] * s[:k]) @ V[:, :k].conj().T).max() < 1e-11
    assert abs(te - float((s[k:] ** 2).sum())) < 1e-13


@pytest.mark.parametrize("direction", ["R", "L"])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 65, 255, 256, 257, 300])
def test_warm_split_orders(k, direction):
    m, n = k + 70, k + 81
    rng = np.random.default_rng(k)
    r = min(m, n)
    U, _ = np.linalg.qr(rng.standard_normal((m, r)))
    V, _ = np.linalg.qr(rng.standard_normal((n, r)))
    s = np.concatenate([np.logspace(0, -3, k), 1e-6 * np.logspace(0, -3, r - k)])
    M = (U * s) @ V.T
    if direction == "R":
        warm = np.linalg.qr(V[:, :k] + 1e-5 * rng.standard_normal((n, k)))[0].T.copy()
    else:
        warm = np.linalg.qr(U[:, :k] + 1e-5 * rng.standard_normal((m, k)))[0].copy()
    left, right, te = dmrg2.warm_split(M, warm, k, direction)
    iso = left.T @ left if direction == "R" else right @ right.T
    assert np.abs(iso - np.eye(k)).max() < 1e-12
    # the kept space is that of the first k pairs to the leak (1e-5) times (s_{k+1}/s_k)^2 per step
    assert np.abs(left @ right - (U[:, :k] * s[:k]) @ V[:, :k].T).max() < 1e-9
    assert abs(te - float((s[k:] ** 2).sum())) < 1e-12
