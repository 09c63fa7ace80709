"""Kernels of the library may start while the kernel before them still runs (programmatic launches): imports over
operands the previous GEMM reads, GEMMs over operands the previous import writes, with no host synchronisation
between them, on the default stream, on a created one and hopping between both.  Every result is kept and compared."""
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


@pytest.mark.parametrize("case", [(700, 1500, 600, 3, "u", 2, "s"), (600, 1030, 520, 8, "s", 8, "s"),
                                  (96, 2000, 200, 4, "s", 1, "b"), (8, 8192, 8, 1, "u", 1, "u"),
                                  (300, 4096, 1, 2, "u", 2, "u")])
@pytest.mark.parametrize("streams", ["default", "created", "both"])
def test_back_to_back(case, streams):
    import torch
    M, K, N, wa, ea, wb, eb = case
    ops = [(datagen.operand(datagen.SEED_BASE + 601 + i, M, K, wa, ea),
            datagen.operand(datagen.SEED_BASE + 701 + i, N, K, wb, eb)) for i in range(3)]
    dev = [(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()) for a, b in ops]
    want = [(b.astype(np.float64) @ a.astype(np.float64).T).astype(np.int64).astype(np.int32) for a, b in ops]
    reps = 24
    outs = torch.zeros(reps, N, M, dtype=torch.int32, device="cuda")
    ctx = allocGEMMContext(M, K, N, wa, wb, ea != "u", eb != "u")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        for r in range(reps):
            a, b = dev[r % 3]
            use = torch.cuda.default_stream() if streams == "default" or (streams == "both" and r % 2) else side
            other = side if use is not side else torch.cuda.default_stream()
            if streams == "both":
                use.wait_stream(other)
            with torch.cuda.stream(use):
                ctx.lhs.importRegular(a)
                ctx.rhs.importRegular(b)
                gemmBitSerial(ctx, out=outs[r])
        torch.cuda.synchronize()
        got = outs.cpu().numpy()
        for r in range(reps):
            assert np.array_equal(got[r], want[r % 3]), r
    finally:
        deallocGEMMContext(ctx)
