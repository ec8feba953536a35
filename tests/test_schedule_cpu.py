"""The factorisation's launches on four streams, replayed on the host: every form
(FP64, integer-digit updates from a threshold and wherever they fit, tensor-core
updates) is free of races, the fronts' memory and the digit slab among them, and
the replay finds each join that is left out, wherever there is a launch that it is for."""
import numpy as np
import pytest

import sam_lib_b200 as spr
from dense_structure import dense_chain

FAR, AHEAD, SLAB, WRITEBACK, SMALL = 1, 2, 4, 8, 16
FORMS = [(0, np.inf), (0, 1e9), (0, 0.0), (1, np.inf)]


def _replay(structure, mixed, least, skip):
    out = np.zeros(4)
    f = spr.load(8).spr_b200_schedule_replay
    import ctypes as C
    f.argtypes = [C.c_void_p] * 3 + [C.c_int, C.c_double, C.c_int, C.c_void_p]
    assert f(*(spr._ptr(a) for a in structure), mixed, least, skip, spr._ptr(out)) == 0
    return [int(v) for v in out]


def _mesh(n):
    from sam_lib_b200.system import load_structure
    st = load_structure(n)
    return st['mspar'], st['mtrees'], st['msifa']


def _retained(widths):
    mspar, mtrees, msifa = dense_chain(widths)
    mspar[56] = 1
    m = len(widths)
    mtrees[mspar[45] - 1 + m + 1 + m - 1] = 1            # SUPSUP of the last supernode
    return mspar, mtrees, msifa


@pytest.mark.parametrize('mixed,least', FORMS)
@pytest.mark.parametrize('n', [4, 9, 12, 16, 24, 32, 48])
def test_meshes(n, mixed, least):
    structure = _mesh(n)
    bad, shared, reused, beside = _replay(structure, mixed, least, 0)
    assert bad == 0
    if reused and n >= 12:
        assert _replay(structure, mixed, least, WRITEBACK)[0] > 0
    if beside:
        assert _replay(structure, mixed, least, SMALL)[0] > 0
    if shared:
        assert _replay(structure, mixed, least, SLAB)[0] > 0
    if n >= 24:
        assert reused and beside
        assert _replay(structure, mixed, least, FAR)[0] > 0 and _replay(structure, mixed, least, AHEAD)[0] > 0
        assert (shared > 0) == (least < np.inf)


@pytest.mark.parametrize('mixed,least', FORMS)
@pytest.mark.parametrize('widths', [[1], [100, 90], [200, 300, 70], [1700, 1080, 50], [2100, 1100]])
@pytest.mark.parametrize('build', [dense_chain, _retained])
def test_chains(build, widths, mixed, least):
    structure = build(widths)
    assert _replay(structure, mixed, least, 0)[0] == 0
