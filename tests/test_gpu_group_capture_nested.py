"""gbs_group_capture on a stream that is already being captured is refused before anything else happens: the caller's
capture goes on, and the graph the group captured before still replays."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext
from gemmbitserial_gb300.grouped import Group

pytestmark = pytest.mark.gpu


def test_refused_inside_a_capture(gbs_lib):
    import torch
    M, K, N = 40, 363, 90
    A = [datagen.operand(datagen.SEED_BASE + 1501 + i, M, K, 2, "u") for i in range(2)]
    B = datagen.operand(datagen.SEED_BASE + 1511, N, K, 2, "s")
    want = [(B.astype(np.int64) @ a.astype(np.int64).T).astype(np.int32) for a in A]
    a0, a1, b = (torch.from_numpy(x).cuda() for x in (*A, B))
    ctx = allocGEMMContext(M, K, N, 2, 2, False, True)
    grp = Group([ctx])
    s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    try:
        grp.capture([a0], [b], stream=s)
        with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):
            x.add_(1)
            with pytest.raises(_capi.GBSError):
                grp.capture([a1], [b], stream=s)
            x.add_(1)
        graph.replay()
        torch.cuda.synchronize()
        assert bool((x == 2).all())
        grp.replay(stream=s)
        torch.cuda.synchronize()
        assert np.array_equal(ctx.res.reshape(N, M), want[0])
        grp.capture([a1], [b], stream=s)
        grp.replay(stream=s)
        torch.cuda.synchronize()
        assert np.array_equal(ctx.res.reshape(N, M), want[1])
    finally:
        grp.free()
        deallocGEMMContext(ctx)
