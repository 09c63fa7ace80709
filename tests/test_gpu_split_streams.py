"""GEMMs of one imported context in flight on several streams, or replayed from a graph beside a live one, into
buffers of their own: few tiles and a long K, where the K split over independent SM pairs keeps partial columns in the
context.  One stream holds that workspace at a time, the others split inside clusters.  Bit-exact against int64."""
import ctypes as C

import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


def operands(M, K, N, seed):
    import torch
    A = datagen.operand(datagen.SEED_BASE + seed, M, K, 2, "u")
    B = datagen.operand(datagen.SEED_BASE + seed + 1, N, K, 2, "s")
    want = (B.astype(np.float64) @ A.astype(np.float64).T).astype(np.int64).astype(np.int32)
    return torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), want


def context(M, K, N):
    ctx = allocGEMMContext(M, K, N, 2, 2, False, True)
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    return ctx


def workspace_splits(ctx, splits):
    """Whether the context's last GEMM split K over `splits` independent pairs."""
    bn, sp, kind = C.c_int(), C.c_int(), C.c_int()
    _capi.check(_capi.load().gbs_debug_last_pair(ctx._h, C.byref(bn), C.byref(sp), C.byref(kind)))
    return (bn.value, sp.value, kind.value) == (256, splits, 0)


@pytest.mark.parametrize("case", [(256, 9216, 4096, 4), (300, 16384, 1300, 4)], ids=lambda c: "x".join(map(str, c[:3])))
def test_one_context_on_two_streams(case):
    import torch
    M, K, N, splits = case
    a, b, want = operands(M, K, N, 1101)
    a2, _, _ = operands(M, K, N, 1111)
    want2 = (b.double() @ a2.double().T).to(torch.int32).cpu().numpy()
    ctx, reps = context(M, K, N), 12
    out = [torch.zeros(reps, N, M, dtype=torch.int32, device="cuda") for _ in range(2)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    try:
        ctx.lhs.importRegular(a)
        ctx.rhs.importRegular(b)
        for lhs, expected, first in ((a, want, 0), (a2, want2, 1)):  # an import gives the workspace back
            torch.cuda.synchronize()
            ctx.lhs.importRegular(lhs, stream=streams[first])
            torch.cuda.synchronize()
            for r in range(reps):
                for i in (first, 1 - first):
                    gemmBitSerial(ctx, stream=streams[i], out=out[i][r])
                    assert workspace_splits(ctx, splits) == (i == first)
            torch.cuda.synchronize()
            for o in out:
                got = o.cpu().numpy()
                for r in range(reps):
                    assert np.array_equal(got[r], expected), r
                o.zero_()
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)


def test_graph_replay_beside_a_live_gemm():
    import torch
    M, K, N, splits = 256, 9216, 4096, 4
    a, b, want = operands(M, K, N, 1121)
    ctx, reps = context(M, K, N), 12
    live, held = torch.cuda.Stream(), torch.cuda.Stream()
    out = torch.zeros(reps, N, M, dtype=torch.int32, device="cuda")
    replayed = torch.zeros(N, M, dtype=torch.int32, device="cuda")
    graph = torch.cuda.CUDAGraph()
    try:
        ctx.lhs.importRegular(a)
        ctx.rhs.importRegular(b)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=held):
            gemmBitSerial(ctx, out=replayed)
        assert not workspace_splits(ctx, splits)
        torch.cuda.synchronize()
        for r in range(reps):
            gemmBitSerial(ctx, stream=live, out=out[r])
            assert workspace_splits(ctx, splits)
            with torch.cuda.stream(held):
                graph.replay()
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        for r in range(reps):
            assert np.array_equal(got[r], want), r
        assert np.array_equal(replayed.cpu().numpy(), want)
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)
