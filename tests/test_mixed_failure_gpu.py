"""A pivot that fails in the mixed-precision mode while the columns beyond the next
super-panel of its own front are being updated on the tensor cores, beside the
panel chain: the outcome is the failing equation, not a wait that ran out.

Rows at - 1 and at are ( 1 1 ; 1 1 ) and zero elsewhere: the pivot is zero in TF32 as
in FP64, so the equation, LIERR, NUMNEG and TOL(2:3) are exact."""
import pytest

from dense_structure import dense_chain, pack_dense
from test_int_update_failure_gpu import _matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('at', [513, 600, 1023, 1025, 1500, 2047, 2900])
def test_a_pivot_that_fails_beside_the_far_update(at):
    import torch
    import sam_lib_b200 as spr
    structure = dense_chain([3000, 1100])
    a = _matrix(4100, at, at)
    d_sm0 = torch.from_numpy(pack_dense(a, *structure)).cuda()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ds = spr.DeviceSolver(*structure)
        ds.set_stream(stream.cuda_stream)
        ds.set_mode(1)
        for guard in (0.0, 0.0, 1e-3):
            ds.set_inertia_guard(guard)
            r = ds.factor(d_sm0.clone())
            assert r['lierr'] == -30 and r['supeqt'] == at + 1
            assert r['numneg'] == int((a.diagonal()[:at] < 0).sum())
            assert r['tol2'] == 0.0 and r['tol3'] == 1.0
            assert ds.info()['fp64_redo'] == (guard > 0.0)
        ds.close()
