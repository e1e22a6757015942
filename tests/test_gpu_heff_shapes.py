"""H_eff at the edges of its dispatch: the one-launch kernel (ragged blocks of rows, empty parts
of the last columns, every 16-row tile count, split contractions) and the tiled contractions
beyond it, dense and sparse MPOs, against numpy.

Each output is a sum of cL Dl d^2 Dr cR products in three stages; with inputs of unit size the
rounding error stays below eps (cL + Dl d^2 + Dr cR) of the result's scale.
"""
import numpy as np
import pytest

import dmrg2

pytestmark = pytest.mark.gpu


def _ref(L, R, WL, WR, th):
    x = np.tensordot(L, th, axes=(2, 0))                     # a w s r e
    ww = np.einsum("wmsp,mnrq->wsrpqn", WL, WR)
    x = np.tensordot(x, ww, axes=((1, 2, 3), (0, 1, 2)))     # a e p q n
    return np.tensordot(x, R, axes=((1, 4), (2, 1)))         # a p q f


SHAPES = [
    (1, 1, 2, 1, 1, 1), (1, 2, 2, 1, 5, 5), (2, 1, 2, 5, 5, 1), (3, 7, 2, 5, 5, 5), (16, 9, 2, 5, 5, 5),
    (17, 33, 2, 8, 8, 8), (33, 40, 2, 1, 3, 8), (64, 64, 2, 5, 5, 5), (50, 129, 2, 5, 5, 5), (130, 100, 2, 5, 5, 5),
    (5, 6, 3, 4, 4, 4), (30, 25, 3, 4, 4, 4), (20, 18, 5, 4, 4, 4), (9, 40, 2, 16, 3, 16), (4, 6, 2, 17, 2, 17),
    (2, 3, 8, 2, 2, 2), (171, 187, 2, 8, 8, 8),
]


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_heff_matches_numpy(shape, sparse, cplx):
    cL, cR, d, Dl, Dm, Dr = shape
    rng = np.random.default_rng(11)

    def rnd(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    L, R, WL, WR, th = rnd(cL, Dl, cL), rnd(cR, Dr, cR), rnd(Dl, Dm, d, d), rnd(Dm, Dr, d, d), rnd(cL, d, d, cR)
    if sparse:
        WL *= rng.random(WL.shape) < 0.2
        WR *= rng.random(WR.shape) < 0.2
    ref = _ref(L, R, WL, WR, th)
    out = dmrg2.apply_heff(L, R, WL, WR, th)
    scale = max(np.abs(ref).max(), 1e-300)
    assert np.abs(out - ref).max() <= 2.3e-16 * (cL + Dl * d * d + Dr * cR) * scale
