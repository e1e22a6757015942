"""A Lanczos solve that leaves no result ends the sweep before its bond's sites are written.

In sweeps without restarts the split is enqueued behind the solve, and the host reads both reports after one
wait. A failure is planted in one such solve (what a barrier that gave up leaves: the solve's flag,
everything else as usual); the call must fail with the numeric status, the sites of that bond and all
behind it must be what they were, and the engine must go on from a fresh state as if nothing had been.
"""
import numpy as np
import pytest

import dmrg2
from dmrg2 import models

from internal import load

pytestmark = pytest.mark.gpu
L, CHI = 10, 12


def _engine(model, **kw):
    cplx = model == "josephson"
    d = 3 if cplx else 2
    mpo = models.josephson(L, n_max=1, E_J=2.0, E_C=1.0, n_g=0.25, phi=0.1) if cplx else models.xxz(L, delta=0.9)
    dt = np.complex128 if cplx else np.float64
    g = dmrg2.DMRG2GPU(L, d, CHI, dtype=dt, krylov_max=30, cutoff=1e-12, tol=1e-300, min_sweeps=10 ** 6, **kw)
    g.set_mpo(mpo)
    g.set_mps(models.random_mps(L, d, CHI, seed=2, dtype=dt))
    return g


def _fail(g, bond, call):
    load().probe_fail_solve(bond + 1)
    with pytest.raises(dmrg2.Dmrg2Error, match="terminate") as e:
        call([CHI])
    assert f"status {dmrg2.ERR_NUMERIC}" in str(e.value)
    return g.get_mps()


def _same(a, b, first):
    for i in range(first, L):
        assert a[i].shape == b[i].shape and np.array_equal(a[i], b[i]), i


def _goes_on(g, start, model, kw):
    """The next run is that of an engine that never failed."""
    twin = _engine(model, **kw)
    for h in (g, twin):
        h.set_mps(start)
        h.run(schedule=[CHI] * 3)
    assert abs(g.get_energy() - twin.get_energy()) <= 1e-12 * abs(twin.get_energy())


@pytest.mark.parametrize("model", ["xxz", "josephson"])
@pytest.mark.parametrize("bond", [0, 4, 6])
def test_failed_solve_before_a_warm_split(model, bond):
    g = _engine(model)
    start = g.get_mps()
    g.run(schedule=[CHI] * 5)
    before = g.get_mps()
    _same(_fail(g, bond, g.resume), before, 0 if bond == 0 else bond + 1)
    _goes_on(g, start, model, {})


@pytest.mark.parametrize("model,kw", [("xxz", {}), ("josephson", {}), ("josephson", {"truncation": 2}),
                                      ("xxz", {"svd_method": 1})])
@pytest.mark.parametrize("bond", [4, 6])
def test_failed_solve_before_the_first_split_at_a_cap(model, kw, bond):
    """The exact, the randomised and the Jacobi split."""
    g = _engine(model, **kw)
    start = g.get_mps()
    run = lambda schedule: (g.set_mps(start), g.run(schedule=schedule))
    for _ in range(3):  # every shape's device loop is captured on its second solve
        run([CHI])
    before = _fail(g, 0, run)  # (canonical; no split has touched the sites from 2 on)
    _same(_fail(g, bond, run), before, bond + 1)
    if kw.get("truncation") != 2:  # (a randomised split's sketch depends on how many the engine has drawn)
        _goes_on(g, start, model, kw)
