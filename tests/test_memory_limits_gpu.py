"""Calls on a device that has no memory left, and the same calls once it has."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = 2 << 20                                    # the device's allocation granularity


class Filler:
    """Takes the device's free memory, some of it in pages of 2 MB."""

    def __init__(self):
        import torch
        torch.cuda.empty_cache()
        self.rt = C.CDLL('libcudart.so.12')
        self.pages = [self._take(PAGE) for _ in range(32)]
        self.blocks = []
        size = 1 << 36
        while size >= PAGE // 16:
            p = self._take(size)
            if p is None:
                size >>= 1
            else:
                self.blocks.append(p)
        self.rt.cudaGetLastError()

    def _take(self, size):
        p = C.c_void_p()
        return p if self.rt.cudaMalloc(C.byref(p), C.c_size_t(size)) == 0 else None

    def give(self, pages):
        for _ in range(pages):
            self.rt.cudaFree(self.pages.pop())

    def close(self):
        for p in self.pages + self.blocks:
            self.rt.cudaFree(p)
        self.pages = self.blocks = []


def _diagonal(neq):
    """Structure of a diagonal matrix: one supernode of one column per equation."""
    one = np.arange(1, neq + 2)
    mtrees = np.concatenate([one, np.ones(neq + 1), np.ones(neq + 1), one, np.zeros(neq), [1, 0]]).astype(np.int64)
    msifa = np.concatenate([one[:-1], one, np.ones(neq), [0]]).astype(np.int64)
    mspar = np.zeros(60, dtype=np.int64)
    mspar[0] = 4
    mspar[2], mspar[3], mspar[7], mspar[10] = len(msifa), len(mtrees), neq, neq
    mspar[12] = mspar[13] = mspar[44] = mspar[46] = 1
    mspar[14] = mspar[15] = neq
    mspar[16] = 3
    mspar[45] = 1 + 3 * (neq + 1)
    mspar[47] = 1 + neq
    return mspar, mtrees, msifa


@pytest.mark.parametrize('pages', [0, 6, 10, 12])
def test_residual_after_an_allocation_that_failed(pages):
    """The residual's row arrays (5, 5 and 2 pages here), none, one, two or all three
    of which fit before the first call gives up."""
    import torch
    import sam_lib_b200 as spr
    neq = 1 << 20
    structure = _diagonal(neq)
    sm = np.concatenate([np.zeros(neq), np.linspace(1.0, 2.0, neq)])
    warm = spr.DeviceSolver(*_diagonal(10))               # the kernels are loaded
    d_w = torch.from_numpy(np.concatenate([np.zeros(10), np.ones(10)])).cuda()
    warm.build_residual(d_w)
    d_sm, d_b = torch.from_numpy(sm).cuda(), torch.ones((1, neq), dtype=torch.float64, device='cuda')
    d_x = torch.empty_like(d_b)
    ds = spr.DeviceSolver(*structure)
    filler = Filler()
    try:
        filler.give(pages)
        with pytest.raises(RuntimeError, match='-4'):
            ds.build_residual(d_sm)
    finally:
        filler.close()
    with pytest.raises(RuntimeError):                     # no matrix yet
        ds.refine(d_sm, d_b, d_x, 1)
    ds.build_residual(d_sm)
    assert ds.factor(d_sm)['lierr'] == 0
    _, berr, _ = ds.refine(d_sm, d_b, d_x, 1, tol=1e-30, maxit=0)
    assert berr <= 1e-15
    assert np.allclose(d_x.cpu().numpy()[0], 1.0 / sm[neq:], rtol=1e-14)
    ds.close()
    warm.close()


@pytest.mark.parametrize('own_stream', [False, True])
def test_solves_take_the_place_of_the_digit_slabs(own_stream):
    """20^3: the factorisation has its digit slabs and nothing is left.  Solves and
    refinement go on, in their place; the factorisation that follows
    does without them, and has them again when there is memory."""
    import contextlib
    import torch
    import sam_lib_b200 as spr
    from sam_lib_b200.system import HexSystem
    hs = HexSystem(20)
    sm = torch.from_numpy(hs.assemble()).cuda()
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream) if own_stream else contextlib.nullcontext():
        b0 = torch.from_numpy(np.random.default_rng(1).uniform(-1.0, 1.0, size=(2, hs.neq))).cuda()
        d, x, y, first = sm.clone(), b0.clone(), torch.empty_like(b0), b0.clone()
        warm = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)   # the kernels are loaded
        ds = spr.DeviceSolver(hs.mspar, hs.mtrees, hs.msifa)
        if own_stream:
            ds.set_stream(stream.cuda_stream)
            warm.set_stream(stream.cuda_stream)
        warm.build_residual(sm)
        warm.factor(d)
        launches = warm.info()['launches']
        warm.solve(d, first, 2)
        warm.close()
        d.copy_(sm)
        assert ds.factor(d)['lierr'] == 0 and ds.info()['launches'] == launches
        ds.build_residual(sm)
        filler = Filler()
        try:
            ds.solve(d, x, 2)                                # the slabs go
            assert torch.equal(x, first)
            d.copy_(sm)
            assert ds.factor(d)['lierr'] == 0
            assert ds.refine(d, b0, y, 2, tol=1e-30, maxit=0)[1] <= 1e-13
            for r in ds.factor(d.copy_(sm)), ds.factor(d.copy_(sm)):
                assert r['lierr'] == 0
        finally:
            filler.close()
        d.copy_(sm)
        assert ds.factor(d)['lierr'] == 0 and ds.info()['launches'] == launches
        x.copy_(b0)
        ds.solve(d, x, 2)
        assert torch.equal(x, first)
        ds.close()
