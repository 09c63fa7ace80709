"""The tensor-core kernel of a context with a side under 256 rows: tile widths and K splits over clusters at their
edges (one stage, stages that do not divide by the split, remainders of rows and columns on either side), results in
a caller's buffer and the context's own.  Bit-exact against int64 products."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu

SHAPES = [(255, 64, 255), (1, 128, 700), (700, 129, 1), (17, 512, 33), (16, 4100, 130), (130, 16384, 16),
          (64, 9216, 300), (384, 2304, 169), (169, 2304, 384), (250, 1000, 4000), (4000, 1111, 3), (5, 16000, 7),
          (128, 8192, 128), (33, 1027, 2050), (200, 600, 20000)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("enc", [(3, "u", 2, "s"), (4, "s", 1, "b")])
def test_small_side(shape, enc):
    import torch
    M, K, N = shape
    wa, ea, wb, eb = enc
    A = datagen.operand(datagen.SEED_BASE + 901, M, K, wa, ea)
    B = datagen.operand(datagen.SEED_BASE + 902, N, K, wb, eb)
    want = (B.astype(np.float64) @ A.astype(np.float64).T).astype(np.int64).astype(np.int32)
    ctx = allocGEMMContext(M, K, N, wa, wb, ea != "u", eb != "u")
    try:
        ctx.set_pipe(_capi.GBS_PIPE_TC)
        assert ctx.pipe == _capi.GBS_PIPE_TC
        ctx.lhs.importRegular(torch.from_numpy(A).cuda())
        ctx.rhs.importRegular(torch.from_numpy(B).cuda())
        out = torch.full((N * M + 64,), 7, dtype=torch.int32, device="cuda")
        for _ in range(3):
            gemmBitSerial(ctx, out=out)
            gemmBitSerial(ctx)
        got = out.cpu().numpy()
        assert np.array_equal(got[:N * M].reshape(N, M), want) and (got[N * M:] == 7).all()
        assert np.array_equal(ctx.res.reshape(N, M), want)
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)
