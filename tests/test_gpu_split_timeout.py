"""A pair of the K-split GEMM whose bounded wait gives up still counts in, so the arrival counters the pairs share end
at zero and the next GEMM of the context is exact.  The wait runs out because nothing was loaded for it: no copy and no
MMA of that pair is in flight, the other pairs run as always."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(256, 9216, 4096), (300, 16384, 270), (2048, 8192, 256), (256, 4000, 9470)],
                         ids=lambda c: "x".join(map(str, c)))
def test_next_gemm_is_exact(gbs_lib, case):
    M, K, N = case
    A = datagen.operand(datagen.SEED_BASE + 1301, M, K, 2, "u")
    B = datagen.operand(datagen.SEED_BASE + 1302, N, K, 2, "s")
    want = (B.astype(np.float64) @ A.astype(np.float64).T).astype(np.int64).astype(np.int32)
    ctx = allocGEMMContext(M, K, N, 2, 2, False, True)
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    try:
        assert gbs_lib.gbs_debug_split_timeout(ctx._h, 64, None) == _capi.GBS_ESTATE  # not imported
        ctx.lhs.importRegular(A)
        ctx.rhs.importRegular(B)
        for _ in range(3):
            assert gbs_lib.gbs_debug_split_timeout(ctx._h, 64, None) == _capi.GBS_ETIMEOUT, gbs_lib.gbs_last_error()
            assert gbs_lib.gbs_debug_tc_error() == 0  # cleared again
            for _ in range(2):
                gemmBitSerial(ctx, stream=0)
                assert np.array_equal(ctx.res.reshape(N, M), want)
        assert gbs_lib.gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)


def test_hook_rejects_what_it_cannot_run(gbs_lib):
    ctx = allocGEMMContext(512, 1024, 512, 2, 2, False, False)
    try:
        ctx.lhs.importRegular(np.zeros((512, 1024), np.int8))
        ctx.rhs.importRegular(np.zeros((512, 1024), np.int8))
        assert gbs_lib.gbs_debug_split_timeout(ctx._h, 64, None) == _capi.GBS_EUNSUPPORTED  # eight stages: no split
        assert gbs_lib.gbs_debug_split_timeout(ctx._h, 0, None) == _capi.GBS_EINVAL
    finally:
        deallocGEMMContext(ctx)
