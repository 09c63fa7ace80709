"""Grouped imports reuse their job table: imports of new tensors back to back on different streams, larger groups of
staged operands, and a captured graph that keeps its own table when imports follow its capture."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext
from gemmbitserial_gb300.grouped import Group

pytestmark = pytest.mark.gpu
DIMS = [(4, 256, 70), (40, 363, 90), (200, 1024, 130), (8, 64, 33)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


def operands(seed):
    """(lhs tensors, rhs tensors, expected results) of every problem."""
    import torch
    ops = [(datagen.operand(seed + 2 * i, M, K, 2, "u"), datagen.operand(seed + 2 * i + 1, N, K, 2, "s"))
           for i, (M, K, N) in enumerate(DIMS)]
    return ([torch.from_numpy(a).cuda() for a, _ in ops], [torch.from_numpy(b).cuda() for _, b in ops],
            [(b.astype(np.int64) @ a.astype(np.int64).T).astype(np.int32) for a, b in ops])


def check(ctxs, want):
    import torch
    torch.cuda.synchronize()
    for c, w in zip(ctxs, want):
        assert np.array_equal(c.res.reshape(w.shape), w)


def test_reimports_and_captured_graph():
    import torch
    ctxs = [allocGEMMContext(M, K, N, 2, 2, False, True) for M, K, N in DIMS]
    grp = Group(ctxs)
    sets = [operands(datagen.SEED_BASE + 800 + 100 * i) for i in range(3)]
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        for r in range(9):  # two streams, ordered by the caller; only the table is shared underneath
            s, other = (s1, s2) if r % 2 else (s2, s1)
            s.wait_stream(other)
            lhs, rhs, want = sets[r % 3]
            grp.import_(lhs, rhs, stream=s)
            grp.gemm(stream=s)
        check(ctxs, sets[8 % 3][2])
        grp.capture(sets[0][0], sets[0][1], stream=s1)
        grp.import_(sets[1][0], sets[1][1])
        grp.gemm()
        check(ctxs, sets[1][2])
        grp.replay()  # the graph still packs the tensors it was captured with
        check(ctxs, sets[0][2])
        grp.capture(sets[2][0], sets[2][1], stream=s2)
        grp.replay()
        check(ctxs, sets[2][2])
        assert grp.status() == _capi.GBS_OK
    finally:
        grp.free()
        for c in ctxs:
            deallocGEMMContext(c)
