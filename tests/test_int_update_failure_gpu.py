"""A pivot that fails while the columns beyond the next super-panel of its own front
are being updated on the integer tensor cores, beside the panel chain: the outcome
is the failing equation, not a wait that ran out.

Rows at - 1 and at of the matrix are ( 1 1 ; 1 1 ) and zero elsewhere, so pivot
`at` is zero; the rest is diagonally dominant with pivots of both signs.  The
equation, LIERR, NUMNEG and TOL(3) = a_jj are exact; the pivot is the rounding of zero."""
import math

import numpy as np
import pytest

from dense_structure import dense_chain, pack_dense

pytestmark = pytest.mark.gpu


def _matrix(neq, seed, at, negative=0.3):
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, size=(neq, neq)) / neq
    a = (a + a.T) / 2
    np.fill_diagonal(a, np.where(rng.random(neq) < negative, -1.0, 1.0))
    a[at - 1: at + 1, :] = a[:, at - 1: at + 1] = 0.0
    a[at - 1: at + 1, at - 1: at + 1] = 1.0
    return a


@pytest.mark.parametrize('at', [513, 560, 600, 1023, 1025, 1100, 1599, 1700, 2098])
def test_a_pivot_that_fails_beside_the_far_update(at):
    import torch
    import sam_lib_b200 as spr
    structure = dense_chain([2100, 1100])
    neq = 3200
    a = _matrix(neq, at, at)
    d_sm0 = torch.from_numpy(pack_dense(a, *structure)).cuda()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ds = spr.DeviceSolver(*structure)
        ds.set_stream(stream.cuda_stream)
        for least in (0.0, math.inf, 0.0, 0.0):
            ds.set_int_min(least)
            r = ds.factor(d_sm0.clone())
            assert r['lierr'] == -30 and r['supeqt'] == at + 1
            assert r['numneg'] == int((a.diagonal()[:at] < 0).sum())
            assert abs(r['tol2']) <= 1e-12 and r['tol3'] == 1.0
        ds.close()


@pytest.mark.parametrize('at', [600, 1500])
def test_the_cholesky_form_stops_at_a_negative_pivot(at):
    """SPRFC2: the matrix is positive definite but for row `at`."""
    import sam_lib_b200 as spr
    mspar, mtrees, msifa = dense_chain([2100, 1100])
    a = _matrix(3200, at, at, negative=0.0)
    a[at - 1, at] = a[at, at - 1] = 0.0
    a[at, at] = -1.0
    sm, tol, msp = pack_dense(a, mspar, mtrees, msifa), np.array([1e-12, 0.0, 0.0]), mspar.copy()
    assert spr.sprfc2(msp, mtrees, msifa, sm, tol) == -3
    assert abs(msp[26]) == at + 1 and tol[1] == -1.0 and tol[2] == -1.0
    spr.release_all()
