"""First uses of a context inside a caller's stream capture: an import whose digit matrix does not exist yet, row- and
column-major and under every capture mode, and the GEMM of a 5-8-bit context that has not run before.  The capture goes
on, and every replay works on the sources as they are then.  Bit-exact against int64."""
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


def product(a, b):
    return (b.astype(np.int64) @ a.astype(np.int64).T).astype(np.int32)


@pytest.mark.parametrize("mode", ["relaxed", "thread_local", "global"])
@pytest.mark.parametrize("col_major", [False, True])
def test_import_captured_first(mode, col_major):
    import torch
    M, K, N = 384, 700, 169
    A = [datagen.operand(datagen.SEED_BASE + 1601 + i, M, K, 2, "u") for i in range(2)]
    B = datagen.operand(datagen.SEED_BASE + 1611, N, K, 2, "u")
    dev = [torch.from_numpy(np.ascontiguousarray(a.T if col_major else a)).cuda() for a in A]
    src, s, graph = torch.zeros_like(dev[0]), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    ctx = allocGEMMContext(M, K, N, 2, 2, False, False)
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    try:
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s, capture_error_mode=mode):
            ctx.lhs.importRegular(src, col_major)
        ctx.rhs.importRegular(torch.from_numpy(B).cuda())
        torch.cuda.synchronize()
        for a, d in zip(A, dev):
            src.copy_(d)
            graph.replay()
            gemmBitSerial(ctx)
            assert np.array_equal(ctx.res.reshape(N, M), product(a, B))
    finally:
        deallocGEMMContext(ctx)


@pytest.mark.parametrize("case", [(64, 500, 300), (300, 700, 260)], ids=lambda c: "x".join(map(str, c)))
def test_wide_gemm_captured_first(case):
    import torch
    M, K, N = case
    A = datagen.operand(datagen.SEED_BASE + 1621, M, K, 8, "s")
    B = datagen.operand(datagen.SEED_BASE + 1622, N, K, 8, "s")
    a, b, graph = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), torch.cuda.CUDAGraph()
    ctx = allocGEMMContext(M, K, N, 8, 8, True, True)
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    out = torch.zeros(N, M, dtype=torch.int32, device="cuda")
    try:
        ctx.lhs.importRegular(a)
        ctx.rhs.importRegular(b)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=torch.cuda.Stream(), capture_error_mode="relaxed"):
            gemmBitSerial(ctx, out=out)
        for _ in range(2):
            out.zero_()
            graph.replay()
            assert np.array_equal(out.cpu().numpy(), product(A, B))
    finally:
        deallocGEMMContext(ctx)
