"""H_eff at the edges of its dispatch: the one-launch kernel (ragged blocks of rows, empty parts
of the last columns, every 16-row tile count, split contractions) and the tiled contractions
beyond it, dense and sparse MPOs, against numpy.

Each output is a sum of cL Dl d^2 Dr cR products in three stages; with inputs of unit size the
rounding error stays below eps (cL + Dl d^2 + Dr cR) of the result's scale.
"""
import ctypes

import numpy as np
import pytest

import dmrg2

from internal import load, ptr

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


@pytest.mark.parametrize("shape,cplx", [((16, 9, 2, 5, 5, 5), False), ((17, 33, 2, 8, 8, 8), True),
                                        ((128, 128, 5, 4, 4, 4), True), ((160, 150, 3, 8, 8, 8), False)])
def test_zeros_of_a_sparse_mpo(shape, cplx):
    """The forms that go over the MPO's nonzeros treat its zeros as the dense product does: an entry
    whose square underflows counts, and an infinity times a zero is NaN in every output it meets."""
    import torch
    cL, cR, d, Dl, Dm, Dr = shape
    rng = np.random.default_rng(12)
    dt = np.complex128 if cplx else np.float64
    L, R, WL, WR, th = (rng.standard_normal(s).astype(dt) for s in (
        (cL, Dl, cL), (cR, Dr, cR), (Dl, Dm, d, d), (Dm, Dr, d, d), (cL, d, d, cR)))
    WL *= (rng.random(WL.shape) < 0.15) * 1e-100
    WR *= (rng.random(WR.shape) < 0.15) * 1e-100

    def run(th):
        t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (L, R, WL, WR, th)]
        out = torch.empty_like(t[4])
        rc = dmrg2.load_library().dmrg2_op_heff_noalloc(
            dmrg2.C128 if cplx else dmrg2.F64, *shape, *[ctypes.c_void_p(x.data_ptr()) for x in (*t, out)],
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        return out.cpu().numpy()

    ref = _ref(L, R, WL * 1e100, WR * 1e100, th)
    out = run(th) * 1e100 * 1e100
    assert np.abs(out - ref).max() <= 2.3e-16 * (cL + Dl * d * d + Dr * cR + 4) * np.abs(ref).max()
    th[cL // 2, 0, d - 1, cR - 1] = np.inf
    assert not np.isfinite(run(th)).any()


@pytest.mark.parametrize("shape,cplx", [((16, 24, 2, 5, 5, 5), False), ((64, 64, 2, 5, 5, 5), False),
                                        ((30, 25, 3, 4, 4, 4), True), ((96, 90, 2, 5, 5, 5), False),
                                        ((64, 64, 5, 4, 4, 4), True)])
@pytest.mark.parametrize("where", ["theta", "shifted", "L"])
def test_out_may_overlap_theta_or_the_left_environment(shape, cplx, where):
    """The one-launch form writes rows of the result while other clusters still read the operands, so
    calls whose result overlaps them take the tiled contractions, at every size."""
    import torch
    cL, cR, d, Dl, Dm, Dr = shape
    rng = np.random.default_rng(13)
    dt = np.complex128 if cplx else np.float64

    def rnd(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    L, R, WL, WR, th = rnd(cL, Dl, cL), rnd(cR, Dr, cR), rnd(Dl, Dm, d, d), rnd(Dm, Dr, d, d), rnd(cL, d, d, cR)
    ref = _ref(L, R, WL, WR, th)
    n = th.size
    # one buffer: [left environment | theta | room for a shifted result]
    buf = torch.from_numpy(np.concatenate([L.ravel(), th.ravel(), np.zeros(n, dt)])).cuda()
    Rd, WLd, WRd = (torch.from_numpy(x).cuda() for x in (R, WL, WR))
    at_th = L.size
    # (two elements further keeps 16-byte alignment)
    at_out = {"theta": at_th, "shifted": at_th + 2, "L": 0}[where]
    ptr = [ctypes.c_void_p(x) for x in (buf.data_ptr(), Rd.data_ptr(), WLd.data_ptr(), WRd.data_ptr(),
                                        buf[at_th:].data_ptr(), buf[at_out:].data_ptr())]
    rc = dmrg2.load_library().dmrg2_op_heff_noalloc(dmrg2.C128 if cplx else dmrg2.F64, *shape, *ptr,
                                                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    out = buf[at_out:at_out + n].cpu().numpy().reshape(ref.shape)
    assert np.abs(out - ref).max() <= 2.3e-16 * (cL + Dl * d * d + Dr * cR) * np.abs(ref).max()


# (shape, complex, share of each W's entries kept): from 16 to 100 inputs, with the nonzeros staged in shared
# memory and with more than fit there
NONZERO = [((96, 90, 2, 5, 5, 5), False, 0.3), ((61, 67, 2, 5, 5, 5), True, 0.3), ((128, 130, 2, 4, 3, 5), False, 0.4),
           ((70, 66, 5, 1, 4, 1), True, 0.5), ((100, 96, 2, 8, 8, 8), False, 0.2), ((64, 60, 2, 8, 6, 8), True, 0.2),
           ((90, 70, 3, 4, 4, 4), False, 0.3), ((30, 40, 5, 4, 4, 4), True, 0.1), ((30, 40, 5, 4, 4, 4), False, 0.5)]


def _nonzeros(shape, cplx, keep):
    cL, cR, d, Dl, Dm, Dr = shape
    rng = np.random.default_rng(14)

    def rnd(*s):
        x = rng.standard_normal(s)
        return x + 1j * rng.standard_normal(s) if cplx else x

    L, R, WL, WR, th = rnd(cL, Dl, cL), rnd(cR, Dr, cR), rnd(Dl, Dm, d, d), rnd(Dm, Dr, d, d), rnd(cL, d, d, cR)
    WL *= rng.random(WL.shape) < keep
    WR *= rng.random(WR.shape) < keep

    def run(th):
        out, nnz = np.empty_like(th), ctypes.c_int()
        assert load().probe_heff_nonzeros(int(cplx), *shape, *[ptr(x) for x in (L, R, WL, WR, th, out)],
                                          ctypes.byref(nnz)) == 0
        return out, nnz.value

    return run, th, _ref(L, R, WL, WR, th)


@pytest.mark.parametrize("shape,cplx,keep", NONZERO)
def test_nonzero_forms_of_the_tiled_path(shape, cplx, keep):
    cL, cR, d, Dl, Dm, Dr = shape
    run, th, ref = _nonzeros(shape, cplx, keep)
    out, nnz = run(th)
    entries = Dl * d ** 4 * Dr
    assert 0 < nnz < entries and (nnz > 768 or keep < 0.5 or entries < 1000)
    assert np.abs(out - ref).max() <= 2.3e-16 * (cL + Dl * d * d + Dr * cR) * np.abs(ref).max()


@pytest.mark.parametrize("shape,cplx,keep", NONZERO)
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_nonzero_forms_spread_what_is_not_finite(shape, cplx, keep, bad):
    """An infinity times a zero of the MPO is NaN in every output that entry meets, as in the dense product."""
    run, th, _ = _nonzeros(shape, cplx, keep)
    th[shape[0] // 2, 0, shape[2] - 1, shape[1] - 1] = bad
    assert not np.isfinite(run(th)[0]).any()
