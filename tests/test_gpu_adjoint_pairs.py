"""The persistent adjoint kernel: tiles of both gradients dealt over the SM pairs (more tiles than pairs, one
gradient only, either contraction the longer, long tiles and left-over ones split over pairs), row and column
remainders, and outputs that do not start on 32 bytes.  dC holds small integers, so every sum is exact in fp32 and
the gradients must equal the int64 products."""
import ctypes as C

import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


@pytest.mark.parametrize("shape", [(1, 1, 1), (33, 8, 31), (256, 256, 256), (257, 264, 65), (64, 1000, 700),
                                   (2600, 1300, 2100), (900, 2300, 3100), (5000, 777, 40),
                                   (6000, 300, 200), (200, 520, 9000), (4096, 2048, 2048)])
@pytest.mark.parametrize("want", ["both", "dA", "dB"])
def test_exact_gradients(shape, want):
    import torch
    M, K, N = shape
    A = datagen.operand(datagen.SEED_BASE + 501, M, K, 3, "u")
    B = datagen.operand(datagen.SEED_BASE + 502, N, K, 4, "s")
    dC = np.random.default_rng(M + N).integers(-6, 7, (N, M)).astype(np.float32)
    ctx = allocGEMMContext(M, K, N, 3, 4, False, True)
    try:
        ctx.lhs.importRegular(torch.from_numpy(A).cuda())
        ctx.rhs.importRegular(torch.from_numpy(B).cuda())
        d = torch.from_numpy(dC).cuda()
        for off in (0, 4):  # floats past an aligned address: 4 leaves 16-byte alignment only
            bufs = [torch.full((rows * K + 8,), 99.0, device="cuda") for rows in (M, N)]
            ptr = [C.c_void_p(b.data_ptr() + 4 * off) if want in ("both", n) else None
                   for b, n in zip(bufs, ("dA", "dB"))]
            _capi.check(_capi.load().gbs_adjoint(ctx._h, C.c_void_p(d.data_ptr()), ptr[0], ptr[1], None))
            torch.cuda.synchronize()
            exact = (dC.T.astype(np.float64) @ B, dC.astype(np.float64) @ A)
            for b, p, e, rows in zip(bufs, ptr, exact, (M, N)):
                got = b.cpu().numpy()
                if p is None:
                    assert (got == 99.0).all()
                    continue
                assert np.array_equal(got[off:off + rows * K].reshape(rows, K), e)
                assert (got[:off] == 99.0).all() and (got[off + rows * K:] == 99.0).all()
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)
