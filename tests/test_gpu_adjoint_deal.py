"""How the adjoint's tiles are dealt where one gradient has few long tiles and the other many short ones (a side of one
to 128 rows against large ones): long tiles whole and in parts, the short ones over the pairs that end first.  dC holds
small integers, so every sum is exact in fp32 and the gradients must equal the products in 64 bits."""
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4096, 4096, 1), (1, 4096, 4096), (4096, 4090, 16), (64, 4096, 4000), (4000, 4096, 128),
                                   (256, 4096, 4096), (1937, 4976, 72), (128, 8192, 2048), (700, 8192, 3), (20000, 700, 2)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("want", ["both", "dA", "dB"])
def test_exact_gradients(gbs_lib, shape, want):
    import torch
    M, K, N = shape
    A = torch.from_numpy(datagen.operand(datagen.SEED_BASE + 1901, M, K, 2, "u")).cuda()
    B = torch.from_numpy(datagen.operand(datagen.SEED_BASE + 1902, N, K, 3, "s")).cuda()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(M + N)
    d = torch.randint(-3, 4, (N, M), generator=gen, device="cuda").float()
    dA, dB = (torch.full((rows, K), 99.0, device="cuda") if want in ("both", n) else None
              for rows, n in ((M, "dA"), (N, "dB")))
    ctx = allocGEMMContext(M, K, N, 2, 3, False, True)
    try:
        ctx.lhs.importRegular(A)
        ctx.rhs.importRegular(B)
        for _ in range(2):
            _capi.check(gbs_lib.gbs_adjoint(ctx._h, d.data_ptr(), *(None if t is None else t.data_ptr() for t in (dA, dB)),
                                            torch.cuda.current_stream().cuda_stream))
        if dA is not None:
            assert torch.equal(dA.double(), d.double().T @ B.double())
        if dB is not None:
            assert torch.equal(dB.double(), d.double() @ A.double())
        assert gbs_lib.gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)
