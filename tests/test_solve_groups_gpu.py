"""Solve sweeps over every way the right-hand sides are grouped (1, 2, groups of
4, pairs of groups, more than a pass takes) and over fronts at the edges of the
64-row blocks and the 256-column tiles of the sweeps.

The check is the normwise backward error of the solution, max|b - K x| /
(||K|| max|x| + max|b|), at most 1e-13 (the bound the residual tests use for an
FP64 factor), and bit equality of one call with its two sweeps called apart."""
import numpy as np
import pytest

from dense_structure import dense_chain, pack_dense

pytestmark = pytest.mark.gpu


def _check(ds, K, d_sm, neq, nrhs, ldb=None):
    import torch
    rng = np.random.default_rng(nrhs)
    ldb = neq if ldb is None else ldb
    b = rng.uniform(-1.0, 1.0, size=(nrhs, ldb))
    x1, x2 = torch.from_numpy(b).cuda(), torch.from_numpy(b).cuda()
    ds.solve(d_sm, x1, nrhs, ldb=ldb)
    ds.solve(d_sm, x2, nrhs, ldb=ldb, which=1)
    ds.solve(d_sm, x2, nrhs, ldb=ldb, which=2)
    assert torch.equal(x1, x2)
    x = x1.cpu().numpy()
    assert np.array_equal(x[:, neq:], b[:, neq:])             # rows beyond NEQ stay
    x, b = x[:, :neq].T, b[:, :neq].T
    r = np.abs(b - K @ x).max(0)
    berr = r / (np.abs(K).sum(1).max() * np.abs(x).max(0) + np.abs(b).max(0))
    assert berr.max() <= 1e-13


@pytest.mark.parametrize('nrhs', [1, 2, 3, 4, 5, 8, 9, 16, 17, 48, 49])
@pytest.mark.parametrize('n', [3, 9, 12])
def test_groups_of_right_hand_sides(n, nrhs):
    import torch
    import sam_lib_b200 as spr
    from sam_lib_b200.system import HexSystem, sm_to_csr
    hs = HexSystem(n)
    sm = hs.assemble()
    K = sm_to_csr(hs.mspar, hs.mtrees, hs.msifa, sm)
    ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
    d_sm = torch.from_numpy(sm).cuda()
    ds.factor(d_sm)
    _check(ds, K, d_sm, hs.neq, nrhs)
    _check(ds, K, d_sm, hs.neq, nrhs, ldb=hs.neq + 3)
    ds.close()


@pytest.mark.parametrize('widths', [[1, 200], [63, 129], [64, 128], [65, 255], [128, 256], [257, 65], [256, 192],
                                    [500, 300, 200], [513, 1]])
@pytest.mark.parametrize('nrhs', [1, 2, 6])
def test_fronts_at_the_tile_edges(widths, nrhs):
    import torch
    import sam_lib_b200 as spr
    structure = dense_chain(widths)
    neq = sum(widths)
    rng = np.random.default_rng(neq)
    a = rng.uniform(-1.0, 1.0, size=(neq, neq)) / neq
    a = (a + a.T) / 2
    np.fill_diagonal(a, np.where(rng.random(neq) < 0.2, -1.0, 1.0))
    ds = spr.DeviceSolver(*structure)
    d_sm = torch.from_numpy(pack_dense(a, *structure)).cuda()
    assert ds.factor(d_sm)['lierr'] == 0
    _check(ds, a, d_sm, neq, nrhs)
    ds.close()


def test_nan_right_hand_sides_end_and_stay_in_their_column():
    """A NaN of any payload (all bits set among them) goes through both sweeps."""
    import torch
    import sam_lib_b200 as spr
    from sam_lib_b200.system import HexSystem
    hs = HexSystem(9)
    ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
    d_sm = torch.from_numpy(hs.assemble()).cuda()
    ds.factor(d_sm)
    b = np.random.default_rng(1).uniform(-1.0, 1.0, size=(5, hs.neq))
    clean = torch.from_numpy(b).cuda()
    ds.solve(d_sm, clean, 5)
    b[1, -1] = np.uint64(0xffffffffffffffff).view(np.float64)
    b[3, 0] = np.nan
    d_b = torch.from_numpy(b).cuda()
    ds.solve(d_sm, d_b, 5)
    x = d_b.cpu().numpy()
    assert np.isnan(x[1]).any() and np.isnan(x[3]).any()
    assert np.array_equal(x[[0, 2, 4]], clean.cpu().numpy()[[0, 2, 4]])
    ds.close()
