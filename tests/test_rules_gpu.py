"""The entry points beside SPRFC1's plain case, on structures that need no reference
library: dense chains of supernodes (one CTA fronts, blocked fronts, one whose update
takes the digit form) and the shipped meshes.  SPRFC2, SPRFC3, SPRFC4, partial
factorisations and the sweeps on them against the oracle; PERI2E against the same
solve in the internal order; the streamed factorisation and the split one against
the plain one.

Tolerances as in the parity tests: factor 1e-10 of the largest entry, solutions 1e-9,
integers exact.  The matrices are diagonally dominant, |a_jj| = 1."""
import ctypes as C
import types

import numpy as np
import pytest

import sam_lib_b200 as spr
from dense_structure import dense_chain, pack_dense
from test_oracle import _lib, _sprsol_ldb, retained_info, run_sprfc3, run_sprfc4, run_sprsol

pytestmark = pytest.mark.gpu

CHAINS = [[40], [100, 70], [3, 90, 60], [200], [130, 200], [60, 300, 260, 100], [577, 129], [1000, 1100]]


def _chain(widths, retained=False):
    mspar, mtrees, msifa = dense_chain(widths)
    m = len(widths)
    if retained:
        mspar[56] = 1
        mtrees[mspar[45] - 1 + m + 1 + m - 1] = 1        # SUPSUP of the last supernode
    return types.SimpleNamespace(neq=sum(widths), mspar=mspar, mtrees=mtrees, msifa=msifa)


def _dense(neq, seed, negative=0.0):
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, size=(neq, neq)) / neq
    a = (a + a.T) / 2
    np.fill_diagonal(a, np.where(rng.random(neq) < negative, -1.0, 1.0))
    return a


def _pair(a, at):
    """Rows at - 1 and at: ( 1 1 ; 1 1 ), alone; pivot `at` is zero."""
    a[at - 1: at + 1, :] = a[:, at - 1: at + 1] = 0.0
    a[at - 1: at + 1, at - 1: at + 1] = 1.0


def _pack(a, rs):
    return pack_dense(a, rs.mspar, rs.mtrees, rs.msifa)


def _close(x, y, tol=1e-10):
    return np.abs(x - y).max() <= tol * np.abs(y).max()


def _rhs(neq, nrhs):
    return np.asfortranarray(np.random.default_rng(neq).uniform(-1.0, 1.0, size=(neq, nrhs)))


def _oracle_chol(rs, sm, b, mspar, ldb, steps):
    p = lambda a: a.ctypes.data_as(C.c_void_p)        # noqa: E731
    i = lambda v: C.byref(C.c_int64(int(v)))          # noqa: E731
    sm, b, msp, tol = sm.copy(), b.copy(order='F'), mspar.copy(), np.array([1e-12, 0.0, 0.0])
    iw = np.zeros(int(msp[13]) + int(msp[12]) + 8, dtype=np.int64)
    rw = np.zeros(int(msp[16]) + int(msp[13]) + 8)
    ierr = C.c_int64(0)
    for s in steps:
        if s == 'f':
            _lib().orc_sprfc2_(p(msp), p(rs.mtrees), p(rs.msifa), p(sm), p(tol), p(iw), p(rw), i(-1), C.byref(ierr))
        elif s == 's':
            _lib().orc_sprfs2_(p(msp), p(rs.mtrees), p(rs.msifa), p(sm), p(b), i(ldb), i(b.shape[1]), p(iw), p(rw),
                               i(-1), C.byref(ierr))
        else:
            _lib().orc_sprbs2_(p(msp), p(rs.mtrees), p(rs.msifa), p(sm), p(b), i(ldb), i(b.shape[1]), p(rw), i(-1),
                               C.byref(ierr))
    return ierr.value, msp, sm, b, tol


def _chol(rs, sm, b, mspar, ldb, steps):
    sm, b, msp, tol = sm.copy(), b.copy(order='F'), mspar.copy(), np.array([1e-12, 0.0, 0.0])
    for s in steps:
        if s == 'f':
            ierr = spr.sprfc2(msp, rs.mtrees, rs.msifa, sm, tol)
        elif s == 's':
            ierr = spr.sprfs2(msp, rs.mtrees, rs.msifa, sm, b, ldb, b.shape[1])
        else:
            ierr = spr.sprbs2(msp, rs.mtrees, rs.msifa, sm, b, ldb, b.shape[1])
    return ierr, msp, sm, b, tol


@pytest.fixture(autouse=True)
def _release():
    yield
    spr.release_all()


@pytest.mark.parametrize('widths', CHAINS)
def test_cholesky_form(widths):
    rs = _chain(widths)
    sm, b = _pack(_dense(rs.neq, 1), rs), _rhs(rs.neq, 3)
    for steps in ('f', 'fs', 'fsb'):
        o, g = _oracle_chol(rs, sm, b, rs.mspar, rs.neq, steps), _chol(rs, sm, b, rs.mspar, rs.neq, steps)
        assert g[0] == o[0] == 0 and np.array_equal(g[1], o[1])
        assert _close(g[2], o[2]) and _close(g[3], o[3], 1e-9) and _close(g[4][1:], o[4][1:])


@pytest.mark.parametrize('widths,at', [([100, 70], 5), ([100, 70], 130), ([577, 129], 513), ([1000, 1100], 600),
                                       ([1000, 1100], 1500)])
def test_cholesky_form_of_an_indefinite_matrix(widths, at):
    rs = _chain(widths)
    a = _dense(rs.neq, 2)
    a[at, at] = -1.0
    sm, b = _pack(a, rs), _rhs(rs.neq, 1)
    o, g = _oracle_chol(rs, sm, b, rs.mspar, rs.neq, 'f'), _chol(rs, sm, b, rs.mspar, rs.neq, 'f')
    assert g[0] == o[0] == -3 and np.array_equal(g[1], o[1]) and abs(g[1][26]) == at + 1
    assert g[4][2] == o[4][2] and abs(g[4][1] - o[4][1]) <= 1e-9


@pytest.mark.parametrize('widths,at', [([40], [1, 17, 39]), ([100, 70], [8, 99, 130]), ([200], [63, 65, 199]),
                                       ([577, 129], [64, 513, 576, 600]), ([1000, 1100], [512, 900, 1700])])
def test_replaced_pivots(widths, at):
    """SPRFC3 on a matrix with pivots of both signs, SPRFC4 on a positive one, with
    pivots that are exactly zero.  DCOR(2, j) names the replaced ones; SPRFC3's DCOR(1, j)
    holds every negative pivot, which is as accurate as the factor."""
    rs = _chain(widths)
    for negative, oracle, gpu in ((0.3, run_sprfc3, spr.sprfc3), (0.0, run_sprfc4, spr.sprfc4)):
        a = _dense(rs.neq, 3, negative)
        for k in at:
            _pair(a, k)
        sm = _pack(a, rs)
        o = oracle('orc', rs, sm, 1e-8, 1e-2)
        f, msp, tol, dcor = sm.copy(), rs.mspar.copy(), np.array([1e-8, 0.0, 0.0, 1e-2]), np.full(2 * rs.neq, 7.0)
        assert gpu(msp, rs.mtrees, rs.msifa, f, tol, dcor) == o['ierr'] == -3
        dcor = dcor.reshape(-1, 2)
        assert np.array_equal(msp, o['mspar']) and np.array_equal(dcor[:, 1], o['dcor'][:, 1])
        assert np.array_equal(np.nonzero(dcor[:, 1])[0], at) and _close(dcor, o['dcor'])
        assert _close(f, o['sm']) and _close(tol[1:3], o['tol'][1:3])


@pytest.mark.parametrize('nrhs', [1, 3, 20])
@pytest.mark.parametrize('widths', [[40, 30], [100, 70], [20, 60, 90], [100, 200], [300, 60], [130, 300], [60, 300, 260],
                                    [577, 129], [1000, 1100]])
def test_partial_factorisation(widths, nrhs):
    """The last supernode is retained: its columns hold the Schur complement, the
    forward sweep leaves the condensed load, LDB < NEQ solves for the others."""
    rs = _chain(widths, retained=True)
    first, _ = retained_info(rs)
    a = _dense(rs.neq, 4, 0.3)
    sm, b = _pack(a, rs), _rhs(rs.neq, nrhs)
    o = run_sprsol('orc', rs, sm, b, iop=1)
    f, msp, tol = sm.copy(), rs.mspar.copy(), np.array([1e-12, 0.0, 0.0])
    assert spr.sprsol(1, msp, rs.mtrees, rs.msifa, f, b.copy(order='F'), rs.neq, nrhs, tol) == o['ierr']
    assert np.array_equal(msp, o['mspar']) and _close(f, o['sm']) and _close(tol[1:], o['tol'][1:])
    assert not f[first:rs.neq].any()
    x, m5 = b.copy(order='F'), msp.copy()
    of = run_sprsol('orc', rs, o['sm'], b, iop=5, mspar=o['mspar'])
    assert spr.sprsol(5, m5, rs.mtrees, rs.msifa, f, x, rs.neq, nrhs, tol) == of['ierr']
    assert _close(x, of['b'], 1e-9)
    cond = b[first:] - a[first:, :first] @ np.linalg.solve(a[:first, :first], b[:first])
    assert _close(x[first:], cond, 1e-9)
    bi = np.asfortranarray(b[:first])
    o3 = _sprsol_ldb('orc', rs, sm, bi, rs.mspar, first)
    f, msp, x = sm.copy(), rs.mspar.copy(), bi.copy(order='F')
    assert spr.sprsol(3, msp, rs.mtrees, rs.msifa, f, x, first, nrhs, tol) == o3['ierr']
    assert _close(x, o3['b'], 1e-9)
    # the same two in the Cholesky form
    ap = _dense(rs.neq, 5)
    sm = _pack(ap, rs)
    o, g = _oracle_chol(rs, sm, bi, rs.mspar, first, 'fsb'), _chol(rs, sm, bi, rs.mspar, first, 'fsb')
    assert g[0] == o[0] == 0 and np.array_equal(g[1], o[1]) and _close(g[2], o[2]) and _close(g[3], o[3], 1e-9)


@pytest.mark.parametrize('widths', [[40], [100, 70], [60, 300, 260, 100]])
def test_external_numbering(widths):
    """PERI2E: B in another order than the equations'."""
    rs = _chain(widths)
    sm, b, tol = _pack(_dense(rs.neq, 6, 0.3), rs), _rhs(rs.neq, 5), np.array([1e-12, 0.0, 0.0])
    want, msp = b.copy(order='F'), rs.mspar.copy()
    ierr = spr.sprsol(3, msp, rs.mtrees, rs.msifa, sm.copy(), want, rs.neq, 5, tol)
    peri2e = np.random.default_rng(0).permutation(rs.neq) + 1
    pere2i = np.empty(rs.neq, dtype=np.int64)
    pere2i[peri2e - 1] = np.arange(1, rs.neq + 1)
    ms = rs.mspar.copy()
    msifa = np.concatenate([peri2e, pere2i, rs.msifa[:int(ms[2])]]).astype(np.int64)
    ms[57] = 2
    ms[[46, 47, 2]] += 2 * rs.neq
    x = np.empty_like(b)
    x[peri2e - 1] = b
    assert spr.sprsol(3, ms, rs.mtrees, msifa, sm.copy(), x, rs.neq, 5, tol) == ierr
    assert np.array_equal(x[peri2e - 1], want)


def _pinned(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


@pytest.mark.parametrize('widths,case', [([100, 70], 'plain'), ([60, 300, 260, 100], 'plain'), ([1000, 1100], 'plain'),
                                         ([60, 300, 260, 100], 'zero'), ([60, 300, 260, 100], 'fails'),
                                         ([1000, 1100], 'fails'), ([1200, 300, 50], 'fails late'),
                                         ([60, 300, 260], 'retained'), ([1000, 1100], 'retained')])
def test_streamed_equals_plain(widths, case):
    """Page-locked SM: the copies run beside the factorisation."""
    rs = _chain(widths, retained=case == 'retained')
    a = _dense(rs.neq, 7, 0.3)
    if case == 'zero':
        a[rs.neq - 40, rs.neq - 40] = 0.0
    elif case == 'fails':
        _pair(a, rs.neq // 3)
    elif case == 'fails late':
        _pair(a, rs.neq - 20)
    sm, b = _pack(a, rs), _rhs(rs.neq, 2)
    iop = 1 if case == 'retained' else 3
    res = []
    for f, x in ((_pinned(sm), _pinned(b.T).T), (sm.copy(), b.copy(order='F'))):
        msp, tol = rs.mspar.copy(), np.array([1e-12, 0.0, 0.0])
        ierr = spr.sprsol(iop, msp, rs.mtrees, rs.msifa, f, x, rs.neq, 2, tol)
        res.append((ierr, msp, tol, np.array(f), np.array(x)))
    assert res[0][0] == res[1][0] and (res[0][0] == -3) == (case in ('zero', 'fails', 'fails late'))
    for u, v in zip(res[0][1:], res[1][1:]):
        assert np.array_equal(u, v)


@pytest.mark.parametrize('n,shift,world', [(9, 0.0, 2), (12, 2.5, 3), (16, 0.0, 2), (20, 2.5, 4)])
def test_split_equals_one_engine(n, shift, world):
    import torch
    from sam_lib_b200.split import emulate
    from sam_lib_b200.system import HexSystem, diag_positions, shift_diagonal
    from sam_lib_b200.workloads import lambda1
    hs = HexSystem(n)
    sm = shift_diagonal(hs.assemble(), diag_positions(hs.mspar, hs.mtrees, hs.msifa),
                        hs.to_internal(hs.box.lumped_mass()), shift * lambda1(n))
    b = _rhs(hs.neq, 3)
    ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
    d_sm, d_b = torch.from_numpy(sm).cuda(), torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
    r = ds.factor(d_sm)
    ds.solve(d_sm, d_b, 3)
    out, sm2, x2 = emulate(hs.mspar, hs.mtrees, hs.msifa, sm, b, world)
    assert out['lierr'] == r['lierr'] == 0 and out['numneg'] == r['numneg'] and (r['numneg'] > 0) == (shift > 0)
    assert _close(sm2, d_sm.cpu().numpy(), 1e-13) and _close(x2, d_b.cpu().numpy().T, 1e-12)
    assert abs(out['tol2'] - r['tol2']) <= 1e-13 * abs(r['tol2'])
    assert abs(out['tol3'] - r['tol3']) <= 1e-13 * abs(r['tol3'])
    ds.close()
