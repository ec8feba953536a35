"""Device assembly against a sum in element order: positions with 1, 2, 4 and 8
contributions (one and two batches of loads, full and partly filled), with an
element matrix each and with one matrix scaled.  Products and sums are rounded
one by one in the same order on both sides, so the results are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [3, 6])
@pytest.mark.parametrize('scaled', [False, True])
def test_device_assembly_equals_sums_in_element_order(n, scaled):
    import torch
    from sam_lib_b200.adjoint import ElementOps
    from sam_lib_b200.system import HexSystem, diag_positions
    hs = HexSystem(n)
    rng = np.random.default_rng(n)
    em = rng.uniform(-1.0, 1.0, size=(1 if scaled else hs.box.nel, 24, 24))
    em = em + em.transpose(0, 2, 1)
    scale = rng.uniform(0.1, 1.0, size=hs.box.nel) if scaled else None
    sm = torch.full((hs.neq + hs.nzerol,), np.nan, dtype=torch.float64, device='cuda')
    ElementOps(hs).assemble(sm, torch.from_numpy(em).cuda(),
                            torch.from_numpy(scale).cuda() if scaled else None)
    # the diagonal, and the sorted multiset of all assembled lower entries
    eq = hs.element_equations()
    want = {}
    for e in range(hs.box.nel):
        for j in range(24):
            for i in range(24):
                a, b = int(eq[e, i]), int(eq[e, j])
                if a >= b >= 0:
                    v = scale[e] * em[0, i, j] if scaled else em[e, i, j]
                    want[a, b] = want.get((a, b), 0.0) + v
    got = sm.cpu().numpy()
    diag = got[diag_positions(hs.mspar, hs.mtrees, hs.msifa)]
    assert np.array_equal(diag, [want[a, a] for a in range(hs.neq)])
    assert np.array_equal(np.sort(got[hs.neq:][got[hs.neq:] != 0.0]), np.sort([v for v in want.values() if v != 0.0]))
