"""Elimination of small fronts (one CTA) and of the 64-column diagonal blocks of
large ones, at the edges of the groups of columns and of the sets of rows that a
warp takes, with pivots of both signs, one child, no child and more children
than are looked up at a time, and a zero pivot at the edges of the groups.

The matrices are diagonally dominant, |a_ii| = 1, so elimination does not grow
their entries and |A - L D L'| <= c F 2^-53 for any order of the sums, F the
front's order; c = 8 covers the reciprocal pivots, the panel's product with
the explicit inverse of its diagonal block and the comparison's own product."""
import numpy as np
import pytest

from dense_structure import dense_chain, pack_dense

pytestmark = pytest.mark.gpu


def forest(widths, root):
    """Leaf supernodes of the given widths, each dense, over one root of `root` columns."""
    mspar, _, _ = dense_chain(list(widths) + [root])
    leaves, neq = len(widths), sum(widths) + root
    m = leaves + 1
    xsuper = np.cumsum([1] + list(widths) + [root])
    xsibl = np.concatenate([np.ones(m), [m]])
    sibl = np.concatenate([np.arange(1, m), [1, 1]])[:m + 1]
    top = np.arange(xsuper[leaves], neq + 1)
    rows = [np.concatenate([np.arange(xsuper[j], xsuper[j + 1]), top]) for j in range(leaves)] + [top]
    f, s = np.array([len(r) for r in rows]), np.diff(xsuper)
    xlindx = np.concatenate([[1], 1 + np.cumsum(f)])
    xlnz = np.concatenate([[1], 1 + np.cumsum(f * s - s * (s - 1) // 2)])
    mtrees = np.concatenate([xsuper, xsibl, sibl, xlindx, np.zeros(m), [1, 0]]).astype(np.int64)
    msifa = np.concatenate([np.concatenate(rows), xlnz, np.ones(m), [0]]).astype(np.int64)
    mspar[2], mspar[3], mspar[13], mspar[14], mspar[15] = len(msifa), len(mtrees), f.max(), f.sum(), xlnz[-1] - 1
    mspar[16] = (leaves + 2) * f.max() * (f.max() + 1)
    mspar[47] = 1 + f.sum()
    return mspar, mtrees, msifa, rows, xsuper, xlnz


def _dense(neq, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, size=(neq, neq)) / neq
    a = (a + a.T) / 2
    np.fill_diagonal(a, np.where(rng.random(neq) < 0.3, -1.0, 1.0))
    return a


def _factor(structure, sm):
    import torch
    import sam_lib_b200 as spr
    ds = spr.DeviceSolver(*structure)
    d = torch.from_numpy(sm).cuda()
    r = ds.factor(d)
    ds.close()
    return r, d.cpu().numpy()


def _residual(a, f, rows, xsuper, xlnz):
    neq = len(a)
    low = np.zeros((neq, neq))
    for j, r in enumerate(rows):
        p = neq + int(xlnz[j]) - 1
        for c in range(xsuper[j] - 1, xsuper[j + 1] - 1):
            i = r[r > c] - 1
            low[i, c] = f[p: p + len(i)]
            p += len(i)
    d = low.diagonal().copy()
    np.fill_diagonal(low, 1.0)
    return np.abs(a - (low * d) @ low.T).max()


def _chain(widths):
    structure = dense_chain(widths)
    mspar, mtrees, msifa = structure
    m, neq = len(widths), sum(widths)
    xsuper = mtrees[:m + 1]
    return structure, [np.arange(xsuper[j], neq + 1) for j in range(m)], xsuper, msifa[mspar[47] - 1: mspar[47] + m]


@pytest.mark.parametrize('widths', [[1], [2], [7], [8], [9], [15], [16], [17], [31], [33], [47], [48], [49], [63], [64], [65],
                                    [80], [81], [112], [113], [144], [145], [175], [176],
                                    [1, 1], [1, 175], [16, 32], [16, 33], [17, 31], [3, 45, 16], [100, 76], [5, 20, 151],
                                    [177], [183], [184], [185], [193], [200], [201], [223], [225], [239], [255], [256],
                                    [9, 168], [65, 200], [129, 1], [192, 1], [193, 60], [257, 127], [320, 128], [449, 77],
                                    [511, 130], [512, 64], [513, 1], [577, 63], [640, 129], [641, 65], [1025, 100],
                                    [100, 449, 200]])
def test_orders_at_the_edges_of_the_groups_and_panels(widths):
    structure, rows, xsuper, xlnz = _chain(widths)
    neq = sum(widths)
    a = _dense(neq, neq)
    r, f = _factor(structure, pack_dense(a, *structure))
    assert r['lierr'] == 0 and r['numneg'] == int((a.diagonal() < 0).sum())
    assert _residual(a, f, rows, xsuper, xlnz) <= 8 * neq * 2.0 ** -53


@pytest.mark.parametrize('leaves,width,root', [(2, 1, 1), (3, 17, 20), (31, 2, 9), (32, 2, 40), (33, 3, 50), (70, 1, 159),
                                               (65, 2, 65)])
def test_many_children(leaves, width, root):
    mspar, mtrees, msifa, rows, xsuper, xlnz = forest([width] * leaves, root)
    neq = leaves * width + root
    a = _dense(neq, neq)
    own = np.arange(neq) // width
    own[leaves * width:] = leaves
    a[(own[:, None] != own[None, :]) & (own[:, None] < leaves) & (own[None, :] < leaves)] = 0.0
    sm = np.zeros(neq + int(mspar[15]))
    for j, r in enumerate(rows):
        p = neq + int(xlnz[j]) - 1
        for c in range(xsuper[j] - 1, xsuper[j + 1] - 1):
            i = r[r > c] - 1
            sm[p: p + len(i)] = a[i, c]
            p += len(i)
    r, f = _factor((mspar, mtrees, msifa), sm)
    assert r['lierr'] == 0 and r['numneg'] == int((a.diagonal() < 0).sum())
    assert _residual(a, f, rows, xsuper, xlnz) <= 8 * neq * 2.0 ** -53


@pytest.mark.parametrize('n', [40, 130, 200, 256])
@pytest.mark.parametrize('at', [1, 7, 8, 9, 15, 16, 33])
def test_the_first_zero_pivot_is_named(n, at):
    """Rows at - 1 and at are ( 1 1 ; 1 1 ) and zero elsewhere: pivot `at` is zero."""
    structure, *_ = _chain([n])
    a = _dense(n, n)
    for i in (at, n - 1):                                 # the last pivot fails as well
        a[i - 1: i + 1, :] = a[:, i - 1: i + 1] = 0.0
        a[i - 1: i + 1, i - 1: i + 1] = 1.0
    r, _ = _factor(structure, pack_dense(a, *structure))
    assert r['lierr'] == -30 and r['supeqt'] == at + 1 and abs(r['tol2']) <= 1e-12
    assert r['numneg'] == int((a.diagonal()[:at] < 0).sum())
