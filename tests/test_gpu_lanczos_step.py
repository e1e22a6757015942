"""The Lanczos step kernels at the edges of their launch shapes, against plain numpy Lanczos.

A solve with a zero tolerance and no restart runs exactly krylov_max steps, so its lowest Ritz
pair is that of numpy's Lanczos (full reorthogonalisation, applied twice) from the same vector.
The lengths n = 4 cL cR cover one block, one full cluster and the first length beyond it, the
grid of one block per SM, ragged slices, and (680 x 680) the streaming passes that serve
vectors beyond the step kernel's shared memory.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

import dmrg2

pytestmark = pytest.mark.gpu

STEPS = 8


def _problem(cL, cR, cplx, seed):
    rng = np.random.default_rng(seed)

    def herm(n):
        x = rng.standard_normal((n, n))
        if cplx:
            x = x + 1j * rng.standard_normal((n, n))
        return (x + x.conj().T) / (2.0 * np.sqrt(n))

    L, R = herm(cL)[:, None, :], herm(cR)[:, None, :]
    WL, WR = (herm(2).T[None, None] + 2.0 * np.eye(2) for _ in range(2))
    th = rng.standard_normal((cL, 2, 2, cR))
    if cplx:
        th = th + 1j * rng.standard_normal(th.shape)
    return L, R, WL, WR, th


def _numpy_ritz(L, R, WL, WR, th, steps):
    def H(v):
        x = (L[:, 0] @ v.reshape(L.shape[0], -1)).reshape(th.shape)
        x = np.einsum("sp,asre->apre", WL[0, 0], x)
        x = np.einsum("rq,apre->apqe", WR[0, 0], x)
        return (x.reshape(-1, R.shape[0]) @ R[:, 0].T).ravel()

    V = [th.ravel() / np.linalg.norm(th)]
    al, be = [], []
    for j in range(steps):
        w = H(V[j])
        al.append(np.vdot(V[j], w).real)
        for _ in range(2):
            for v in V:
                w = w - np.vdot(v, w) * v
        be.append(np.linalg.norm(w))
        if j + 1 < steps:
            V.append(w / be[j])
    ev, y = np.linalg.eigh(np.diag(al) + np.diag(be[: steps - 1], 1) + np.diag(be[: steps - 1], -1))
    return ev[0], np.stack(V, 1) @ y[:, 0]


@pytest.mark.parametrize("cL,cR,cplx", [
    (2, 1, False), (8, 16, False), (3, 43, False), (37, 73, False), (64, 128, False), (64, 129, False),
    (256, 256, False), (680, 680, False), (8, 16, True), (64, 64, True), (64, 65, True), (150, 151, True),
])
def test_fixed_number_of_steps_matches_numpy(cL, cR, cplx):
    L, R, WL, WR, th = _problem(cL, cR, cplx, 3)
    steps = min(STEPS, 4 * cL * cR)
    e_ref, v_ref = _numpy_ritz(L, R, WL, WR, th, steps)
    e, v = dmrg2.optimize_two_site(L, R, WL, WR, th, max_iter=steps, tol=0.0, max_restarts=0)
    v = v.ravel()
    assert abs(e - e_ref) <= 1e-13 * max(1.0, np.abs(e_ref)) * steps
    assert abs(np.linalg.norm(v) - 1.0) < 1e-13
    phase = np.vdot(v, v_ref)
    # Ritz coefficients move by rounding over the gap of the small tridiagonal matrix (~0.1)
    assert np.linalg.norm(v * (phase / abs(phase)) - v_ref) < 1e-11


def test_zero_start_is_replaced_by_a_random_vector():
    L, R, WL, WR, th = _problem(40, 60, False, 5)
    e, v = dmrg2.optimize_two_site(L, R, WL, WR, np.zeros_like(th), max_iter=100, tol=1e-12, max_restarts=4)
    ev = [np.linalg.eigvalsh(m) for m in (L[:, 0], WL[0, 0].T, WR[0, 0].T, R[:, 0])]
    best = min(a * b * c * d for a in (ev[0][0], ev[0][-1]) for b in (ev[1][0], ev[1][-1])
               for c in (ev[2][0], ev[2][-1]) for d in (ev[3][0], ev[3][-1]))
    assert abs(e - best) < 1e-9 * abs(best)
    assert abs(np.linalg.norm(v) - 1.0) < 1e-13


CHILD = """
import test_gpu_lanczos_step as t
for case in [(64, 129, False), (100, 101, False), (150, 151, True)]:
    t.test_fixed_number_of_steps_matches_numpy(*case)
print("ok")
"""


@pytest.mark.parametrize("blocks", [0, 17, 60])
def test_fewer_blocks_than_sms(blocks):
    """A context with fewer SMs (a partition of the GPU) runs the cooperative kernels on as many blocks, and
    the streaming passes where there are none."""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, DMRG2_TEST_STEP_BLOCKS=str(blocks), PYTHONPATH=os.pathsep.join([here] + sys.path))
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.split() == ["ok"], r.stderr

