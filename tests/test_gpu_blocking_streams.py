"""The legacy default stream and blocking streams wait for each other without events; the library's programmatic
launches on the default stream keep that.  A blocking stream writes an import's source late, the default stream imports
and multiplies it, the blocking stream reads the result: no synchronisation by the host or by events in between."""
import ctypes as C

import numpy as np
import pytest

from gemmbitserial_gb300 import datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


@pytest.fixture()
def blocking():
    """A stream created without the non-blocking flag (torch's own streams have it)."""
    import torch
    torch.zeros(1, device="cuda")  # the context
    driver, handle = C.CDLL("libcuda.so.1"), C.c_void_p()
    assert driver.cuStreamCreate(C.byref(handle), 0) == 0
    yield torch.cuda.ExternalStream(handle.value)
    torch.cuda.synchronize()
    driver.cuStreamDestroy_v2(handle)


@pytest.mark.parametrize("case", [(8, 8192, 8, 1, "u", 1, "u"), (384, 2304, 169, 2, "u", 2, "u"),
                                  (256, 9216, 1024, 1, "b", 4, "s"), (600, 1030, 520, 8, "s", 8, "s"),
                                  (2048, 4096, 2048, 3, "u", 2, "s")])
def test_default_stream_beside_a_blocking_one(case, blocking):
    import torch
    M, K, N, wa, ea, wb, eb = case
    lhs = [datagen.operand(datagen.SEED_BASE + 1201 + i, M, K, wa, ea) for i in range(3)]
    rhs = datagen.operand(datagen.SEED_BASE + 1211, N, K, wb, eb)
    want = [(rhs.astype(np.float64) @ a.astype(np.float64).T).astype(np.int64).astype(np.int32) for a in lhs]
    versions = [torch.from_numpy(a).cuda() for a in lhs]
    reps = 18
    src = torch.zeros(M, K, dtype=versions[0].dtype, device="cuda")
    out = torch.zeros(N, M, dtype=torch.int32, device="cuda")
    kept = torch.zeros(reps, N, M, dtype=torch.int32, device="cuda")
    ctx = allocGEMMContext(M, K, N, wa, wb, ea != "u", eb != "u")
    try:
        ctx.rhs.importRegular(torch.from_numpy(rhs).cuda())
        torch.cuda.synchronize()
        for r in range(reps):
            with torch.cuda.stream(blocking):
                torch.cuda._sleep(200_000)  # about 100 us
                src.copy_(versions[r % 3])
            ctx.lhs.importRegular(src)
            gemmBitSerial(ctx, out=out)
            with torch.cuda.stream(blocking):
                kept[r].copy_(out)
        torch.cuda.synchronize()
        got = kept.cpu().numpy()
        for r in range(reps):
            assert np.array_equal(got[r], want[r % 3]), r
    finally:
        deallocGEMMContext(ctx)
