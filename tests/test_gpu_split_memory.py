"""A context whose GEMM splits K over independent pairs, with no room for that kernel's workspace behind a digit matrix:
the digit matrix is allocated alone."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", ["import", "gemm"])
def test_digits_without_the_workspace(gbs_lib, at):
    M, K, N = 300, 16384, 270
    A = datagen.operand(datagen.SEED_BASE + 1701, M, K, 2, "u")
    B = datagen.operand(datagen.SEED_BASE + 1702, N, K, 2, "s")
    want = (B.astype(np.float64) @ A.astype(np.float64).T).astype(np.int64).astype(np.int32)
    ctx = allocGEMMContext(M, K, N, 2, 2, False, True)
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    launches = []
    try:
        # an allocation fails: the first of the import (digits and workspace together), or of the first GEMM after
        # imports that wrote planes only
        if at == "gemm":
            ctx.set_pipe(_capi.GBS_PIPE_POPC)
        else:
            gbs_lib.gbs_debug_fail_alloc_after(1)
        ctx.lhs.importRegular(A)
        ctx.rhs.importRegular(B)
        ctx.set_pipe(_capi.GBS_PIPE_TC)
        if at == "gemm":
            gbs_lib.gbs_debug_fail_alloc_after(1)
        for _ in range(2):
            before = gbs_lib.gbs_debug_launch_count()
            gemmBitSerial(ctx, stream=0)
            launches.append(gbs_lib.gbs_debug_launch_count() - before)
            assert np.array_equal(ctx.res.reshape(N, M), want)
        assert launches[1] == 1 and launches[0] == (1 if at == "import" else 3)  # the digits were there, or expanded
    finally:
        gbs_lib.gbs_debug_fail_alloc_after(0)
        deallocGEMMContext(ctx)
