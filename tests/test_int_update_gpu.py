"""FP64 Schur updates as 8-bit digit products on the integer tensor cores.

Dense fronts whose update sizes fall on and beside the smallest that the digit
form takes (1024 rows, 128 columns), the edges of the 128 x 64 tiles, of the
128-column K blocks and of the 512-column super-panels (odd first columns among
them), with pivots of both signs and rows scaled over
six decades.  The matrices are diagonally dominant (up to the scaling), so
elimination does not grow their entries, and with A = S B S, |B_ii| = 1,

    |A - L D L'|_ij <= c F 2^-53 S_i S_j

for any order of the sums, F the front's order.  The digit form drops less
than 2^-60 S_i S_j per term, far below; c = 8 covers the panel's product with
the explicit inverse of its diagonal block and the comparison's own product."""
import math

import numpy as np
import pytest

from dense_structure import dense_chain, pack_dense
from test_pivot_blocks_gpu import forest

pytestmark = pytest.mark.gpu


def _matrix(neq, seed, negative):
    rng = np.random.default_rng(seed)
    b = rng.uniform(-1.0, 1.0, size=(neq, neq)) / neq
    b = (b + b.T) / 2
    sign = np.where(rng.random(neq) < 0.3, -1.0, 1.0) if negative else np.ones(neq)
    np.fill_diagonal(b, sign)
    s = 10.0 ** rng.uniform(-3.0, 3.0, size=neq)
    return b * s[:, None] * s[None, :], s, int((sign < 0).sum())


def _factor(ds, sm, least):
    import torch
    ds.set_int_min(least)
    d = torch.from_numpy(sm).cuda()
    r = ds.factor(d)
    return r, d.cpu().numpy()


def _unpack(sm, neq, mspar, mtrees, msifa):
    m = int(mspar[10])
    xsuper, xlnz = mtrees[:m + 1], msifa[mspar[47] - 1: mspar[47] + m]
    low = np.zeros((neq, neq))
    for j in range(m):
        p = xlnz[j] - 1 + neq
        for c in range(xsuper[j] - 1, xsuper[j + 1] - 1):
            low[c:, c] = sm[p: p + neq - c]
            p += neq - c
    return low


@pytest.mark.parametrize('negative', [False, True])
@pytest.mark.parametrize('widths', [[128, 1024], [129, 1025], [200, 1087], [255, 1088], [513, 1024], [640, 1089],
                                    [576, 1200], [1025, 130, 1100], [1600, 1027]])
def test_digit_updates_reproduce_the_matrix(widths, negative):
    import sam_lib_b200 as spr
    structure = dense_chain(widths)
    neq = sum(widths)
    a, s, nneg = _matrix(neq, neq, negative)
    sm = pack_dense(a, *structure)
    ds = spr.DeviceSolver(*structure)
    r, f = _factor(ds, sm, 0.0)
    launches = ds.info()['launches']
    rg, fg = _factor(ds, sm, math.inf)                   # the general path
    assert r['lierr'] == rg['lierr'] == 0 and r['numneg'] == rg['numneg'] == nneg
    assert launches > ds.info()['launches']              # a split and a product for each update
    low = _unpack(f, neq, *structure)
    d = low.diagonal().copy()
    np.fill_diagonal(low, 1.0)
    err = np.abs(a - (low * d) @ low.T) / (s[:, None] * s[None, :])
    assert err.max() <= 8 * neq * 2.0 ** -53
    # the two paths' factors: both within the bound of A, and L is as well conditioned as B
    scale = np.sqrt(np.abs(d))[None, :] / s[:, None]
    lg = _unpack(fg, neq, *structure)
    np.fill_diagonal(lg, 1.0)
    assert (np.abs(low - lg) * scale).max() <= 32 * neq * 2.0 ** -53
    ds.close()


def test_levels_with_large_and_small_fronts():
    """16^3: levels whose fronts go partly to the digit form and partly to the
    FP64 kernel; the factor within the parity tests' 1e-10 of the general path's."""
    import sam_lib_b200 as spr
    from sam_lib_b200.system import HexSystem
    hs = HexSystem(16)
    sm = hs.assemble()
    ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
    r, f = _factor(ds, sm, 0.0)
    launches = ds.info()['launches']
    rg, fg = _factor(ds, sm, math.inf)
    assert r['lierr'] == rg['lierr'] == 0 and launches > ds.info()['launches']
    assert np.abs(f - fg).max() <= 1e-10 * np.abs(fg).max()
    ds.close()


def test_far_columns_of_a_small_front_beside_a_large_one():
    """Two fronts of one level in the same panel steps, both with columns beyond
    the next super-panel: after 512 columns one has 1238 rows left (digit
    form), the other 618 (FP64 kernel)."""
    import sam_lib_b200 as spr
    widths, root = [1700, 1080], 50
    own = np.cumsum([0] + widths)
    neq = sum(widths) + root
    structure = forest(widths, root)
    rows, xlnz = structure[3], structure[5]
    structure = structure[:3]
    a, s, nneg = _matrix(neq, 7, True)
    a[own[0]:own[1], own[1]:own[2]] = a[own[1]:own[2], own[0]:own[1]] = 0.0
    starts = np.concatenate([own, [neq]])
    sm = np.zeros(neq + int(structure[0][15]))

    def columns():
        for j, r in enumerate(rows):
            p = neq + int(xlnz[j]) - 1
            for c in range(starts[j], starts[j + 1]):
                i = r[r > c] - 1
                yield c, i, slice(p, p + len(i))
                p += len(i)
    for c, i, at in columns():
        sm[at] = a[i, c]
    ds = spr.DeviceSolver(*structure)
    r, f = _factor(ds, sm, 0.0)
    launches = ds.info()['launches']
    rg, _ = _factor(ds, sm, math.inf)
    assert r['lierr'] == rg['lierr'] == 0 and r['numneg'] == rg['numneg'] == nneg
    assert launches > ds.info()['launches']
    low = np.zeros((neq, neq))
    for c, i, at in columns():
        low[i, c] = f[at]
    d = low.diagonal().copy()
    np.fill_diagonal(low, 1.0)
    err = np.abs(a - (low * d) @ low.T) / (s[:, None] * s[None, :])
    assert err.max() <= 8 * neq * 2.0 ** -53
    ds.close()


def test_nan_fails_at_the_same_equation():
    import sam_lib_b200 as spr
    structure = dense_chain([640, 1024])
    a, _, _ = _matrix(1664, 3, False)
    a[700, 5] = a[5, 700] = math.nan
    sm = pack_dense(a, *structure)
    ds = spr.DeviceSolver(*structure)
    r, _ = _factor(ds, sm, 0.0)
    rg, _ = _factor(ds, sm, math.inf)
    assert r['lierr'] == rg['lierr'] == -30 and r['supeqt'] == rg['supeqt'] == 701
    ds.close()


def test_a_wait_that_runs_out_is_reported():
    import sam_lib_b200 as spr
    import torch
    structure = dense_chain([640, 1024])
    a, _, _ = _matrix(1664, 4, False)
    sm = pack_dense(a, *structure)
    ds = spr.DeviceSolver(*structure)
    ds.set_int_min(0.0)
    ds.set_watchdog(0.05, drop=True)                     # one CTA never loads its first operands
    with pytest.raises(RuntimeError, match='-4'):
        ds.factor(torch.from_numpy(sm).cuda())
    ds.set_watchdog(2.0, drop=False)
    r, f = _factor(ds, sm, 0.0)
    rg, fg = _factor(ds, sm, math.inf)
    assert r['lierr'] == rg['lierr'] == 0 and np.abs(f - fg).max() <= 1e-12 * np.abs(fg).max()
    ds.close()
