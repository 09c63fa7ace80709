"""GEMMs with a side under 256 rows, on either side of what decides their kernel: few tiles and many, short and long K,
lhs rows that align the result's rows and not, the larger side left and right, 1- to 8-bit operands; on device results,
under capture, and again after new imports.  Bit-exact against int64."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu
CASES = [(255, 256, 20001), (20001, 256, 255), (128, 130, 39000), (129, 64, 20000), (16, 1500, 30000), (17, 1500, 30000),
         (30000, 1500, 17), (48, 8000, 5000), (200, 8192, 9000), (9000, 8192, 200), (9, 100, 45001), (100, 8192, 300),
         (300, 8192, 100), (1, 4000, 20000), (33, 1000, 33), (255, 16384, 255)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


def product(a, b):
    import torch
    return (torch.from_numpy(b).cuda().double() @ torch.from_numpy(a).cuda().double().T).to(torch.int32)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c)))
@pytest.mark.parametrize("enc", [(2, "u", 2, "s"), (1, "b", 4, "s"), (8, "s", 3, "u")])
def test_shapes(case, enc):
    import torch
    M, K, N = case
    wa, ea, wb, eb = enc
    if wa == 8 and K * 15 * 7 >= 1 << 24:
        pytest.skip("past the exactness bound of the parts")
    A = [datagen.operand(datagen.SEED_BASE + 1801 + i, M, K, wa, ea) for i in range(2)]
    B = datagen.operand(datagen.SEED_BASE + 1811, N, K, wb, eb)
    want = [product(a, B) for a in A]
    ctx = allocGEMMContext(M, K, N, wa, wb, ea != "u", eb != "u")
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    out, s, graph = torch.zeros(N, M, dtype=torch.int32, device="cuda"), torch.cuda.Stream(), torch.cuda.CUDAGraph()
    try:
        ctx.rhs.importRegular(torch.from_numpy(B).cuda())
        ctx.lhs.importRegular(torch.from_numpy(A[0]).cuda())
        if wa <= 4:  # the first GEMM recorded: no table can be made in a capture
            torch.cuda.synchronize()
            with torch.cuda.graph(graph, stream=s):
                gemmBitSerial(ctx, out=out)
            graph.replay()
            assert torch.equal(out, want[0])
        for i in (0, 1, 0):
            ctx.lhs.importRegular(torch.from_numpy(A[i]).cuda())
            out.zero_()
            gemmBitSerial(ctx, out=out)
            assert torch.equal(out, want[i])
            if wa <= 4:
                out.zero_()
                graph.replay()
                assert torch.equal(out, want[i])
        gemmBitSerial(ctx)
        assert np.array_equal(ctx.res.reshape(N, M), want[0].cpu().numpy())
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)
