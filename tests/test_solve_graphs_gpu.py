"""Solves that are replayed from a graph after the solver's work buffers moved.

A call with more right-hand sides than any before makes the buffers anew; a
graph captured before that holds the old ones.  One handle on a stream of its
own solves with counts that go up and down again, always on the same arrays, and
every result equals, bit for bit, that of a handle that only ever saw the one count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('counts', [[1, 2, 1], [1, 2, 3, 4, 1, 2, 3], [3, 17, 3, 49, 17, 3, 1], [4, 48, 4, 48]])
@pytest.mark.parametrize('n', [6, 12])
def test_counts_that_go_up_and_down(n, counts):
    import torch
    import sam_lib_b200 as spr
    from sam_lib_b200.system import HexSystem
    hs = HexSystem(n)
    b0 = torch.from_numpy(np.random.default_rng(n).uniform(-1.0, 1.0, size=(max(counts), hs.neq))).cuda()
    b = torch.empty_like(b0)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        assembled = torch.from_numpy(hs.assemble()).cuda()
        d_sm = assembled.clone()
        ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
        ds.set_stream(stream.cuda_stream)
        ds.factor(d_sm)
        for nrhs in counts:
            fresh = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
            fresh.set_stream(stream.cuda_stream)
            own, want = assembled.clone(), b0.clone()
            fresh.factor(own)
            fresh.solve(own, want, nrhs)
            fresh.close()
            for _ in range(2):                                # the second pass of a count replays
                b.copy_(b0)
                ds.solve(d_sm, b, nrhs)
                assert torch.equal(b, want)
        ds.close()
