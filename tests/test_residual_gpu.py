"""The residual operator built from SM: rows of any length, against scipy.

A symmetric matrix that fills the whole symbolic pattern (rows of hundreds to
thousands of entries, where an assembled mesh has 81) is compacted, and the
backward error of one solve through it is compared with the one scipy forms
from the same matrix: both are a residual's maximum norm, so the sums' order
leaves at most NEQ roundings between them."""
import numpy as np
import pytest

from sam_lib_b200.system import HexSystem, diag_positions, sm_to_csr


@pytest.mark.gpu
@pytest.mark.parametrize('n, zeros', [(3, 0.0), (5, 0.0), (5, 0.9), (9, 0.5)])
def test_residual_of_a_filled_pattern(n, zeros):
    import torch
    import sam_lib_b200 as spr
    hs = HexSystem(n)
    rng = np.random.default_rng(n)
    sm = np.zeros(hs.neq + hs.nzerol)
    sm[hs.neq:] = rng.uniform(-1.0, 1.0, size=hs.nzerol) * (rng.random(hs.nzerol) >= zeros)
    pos = diag_positions(hs.mspar, hs.mtrees, hs.msifa)
    sm[pos] = 2.0 * hs.neq                                   # diagonally dominant
    K = sm_to_csr(hs.mspar, hs.mtrees, hs.msifa, sm)
    b = rng.uniform(-1.0, 1.0, size=(3, hs.neq))
    ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
    d_sm = torch.from_numpy(sm).cuda()
    ds.build_residual(d_sm)
    ds.build_residual(d_sm)                                  # once more on the kept buffers
    ds.factor(d_sm)
    d_b = torch.from_numpy(b).cuda()
    d_x = torch.empty_like(d_b)
    it, berr, _ = ds.refine(d_sm, d_b, d_x, 3, tol=1e-30, maxit=0)
    x = d_x.cpu().numpy()
    r = np.abs(b.T - K @ x.T).max(0)
    norm = np.abs(K).sum(1).max()
    host = (r / (norm * np.abs(x).max(1) + np.abs(b).max(1))).max()
    # each residual entry is a sum of at most NEQ + 1 terms bounded by norm max|x| + max|b|
    assert it == 0 and abs(host - berr) <= 2 * (hs.neq + 1) * 2.0 ** -53
    assert berr <= 1e-13
    ds.close()
