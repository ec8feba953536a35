"""The residual operator does not depend on the order in which its rows were filled:
the backward error, which is divided by the largest row sum, is the same bit
for bit however often the operator is built."""
import numpy as np
import pytest

from sam_lib_b200.system import HexSystem, diag_positions


@pytest.mark.gpu
@pytest.mark.parametrize('n', [5, 9, 12])
def test_builds_give_the_same_backward_error(n):
    import torch
    import sam_lib_b200 as spr
    hs = HexSystem(n)
    rng = np.random.default_rng(n)
    sm = np.zeros(hs.neq + hs.nzerol)
    sm[hs.neq:] = rng.uniform(-1.0, 1.0, size=hs.nzerol)     # rows of hundreds of entries
    sm[diag_positions(hs.mspar, hs.mtrees, hs.msifa)] = 2.0 * hs.neq
    d_sm = torch.from_numpy(sm).cuda()
    d_b = torch.from_numpy(rng.uniform(-1.0, 1.0, size=(1, hs.neq))).cuda()
    d_x = torch.empty_like(d_b)
    ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
    d_f = d_sm.clone()
    ds.factor(d_f)
    seen = set()
    for _ in range(20):
        ds.build_residual(d_sm)
        seen.add(ds.refine(d_f, d_b, d_x, 1, tol=1e-30, maxit=0)[1])
    assert len(seen) == 1
    ds.close()
