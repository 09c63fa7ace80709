"""The fused kernel of 5-8-bit operands (M, N >= 256): largest values up to the bound where a sum in one of its two
accumulators would leave the exact range, K past it (split over CTAs, odd result sizes among them), every import
form that writes the part digit matrices, and changes between the fused and the separate form.  Against int64."""
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


def cuda(x):
    import torch
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def product(A, B):
    """int32 wrap-around of the exact product (|sum| < 2^53 in float64)."""
    return (B.astype(np.float64) @ A.astype(np.float64).T).astype(np.int64).astype(np.int32)


def operand(seed, rows, K, bits, enc):
    return datagen.operand(datagen.SEED_BASE + seed, rows, K, bits, enc, np.int16)


def run(A, B, wa, ea, wb, eb):
    import torch
    ctx = allocGEMMContext(A.shape[0], A.shape[1], B.shape[0], wa, wb, ea != "u", eb != "u")
    try:
        assert ctx.pipe == _capi.GBS_PIPE_TC
        ctx.lhs.importRegular(cuda(A))
        ctx.rhs.importRegular(cuda(B))
        out = torch.empty(B.shape[0], A.shape[0], dtype=torch.int32, device="cuda")
        gemmBitSerial(ctx, out=out)
        return out.cpu().numpy()
    finally:
        deallocGEMMContext(ctx)


# (wa, ea, va, wb, eb, vb, K): every element at its largest magnitude
@pytest.mark.parametrize("case", [(8, "u", 255, 8, "u", 255, 4096), (8, "u", 255, 8, "u", 255, 4142),
                                  (8, "u", 255, 8, "u", 255, 8200), (8, "s", -128, 8, "s", -128, 13200),
                                  (8, "s", 127, 8, "s", -128, 13300), (5, "u", 31, 8, "u", 255, 4000),
                                  (8, "u", 255, 5, "s", -16, 9000), (8, "u", 255, 4, "u", 15, 60000),
                                  (1, "b", 1, 7, "u", 127, 20000), (6, "s", -32, 2, "u", 3, 5000)])
def test_largest_values(case):
    wa, ea, va, wb, eb, vb, K = case
    A, B = np.full((257, K), va, np.int16), np.full((258, K), vb, np.int16)
    A[::3, ::5] = 0 if ea != "b" else -1  # rows of other sums
    B[::7, ::3] = 1
    assert np.array_equal(run(A, B, wa, ea, wb, eb), product(A, B))
    assert _capi.load().gbs_debug_tc_error() == 0


@pytest.mark.parametrize("shape", [(256, 64, 256), (257, 130, 259), (511, 16000, 301), (1000, 4500, 777)])
@pytest.mark.parametrize("enc", [(8, "u", 8, "u"), (8, "s", 8, "s"), (7, "s", 5, "u"), (5, "s", 6, "s"),
                                 (8, "s", 3, "u"), (2, "s", 6, "u"), (1, "b", 8, "u")])
def test_random_values(shape, enc):
    M, K, N = shape
    wa, ea, wb, eb = enc
    A, B = operand(401, M, K, wa, ea), operand(402, N, K, wb, eb)
    assert np.array_equal(run(A, B, wa, ea, wb, eb), product(A, B))
    assert _capi.load().gbs_debug_tc_error() == 0


def test_import_forms_and_forms_of_the_gemm():
    """Column-major and threshold imports, single-bit writes, and the separate form forced between fused GEMMs."""
    M, K, N = 300, 777, 270
    A, B = operand(403, M, K, 8, "u"), operand(404, N, K, 8, "s")
    ctx = allocGEMMContext(M, K, N, 8, 8, False, True)
    lib = _capi.load()
    try:
        def check():
            gemmBitSerial(ctx)
            assert np.array_equal(ctx.res.reshape(N, M), product(A, B))
        ctx.lhs.importRegular(cuda(A.T), readColMajor=True)
        ctx.rhs.importRegular(cuda(B))
        check()
        _capi.check(lib.gbs_set_variant(ctx._h, 512))  # separate form
        check()
        B = np.ascontiguousarray(B[::-1])
        ctx.rhs.importRegular(cuda(B.T), readColMajor=True)
        check()
        _capi.check(lib.gbs_set_variant(ctx._h, -1))
        check()
        thr = np.sort(np.random.default_rng(5).integers(-3000, 3000, (200, M)).astype(np.int32), axis=0)
        X = np.random.default_rng(6).integers(-3000, 3000, (M, K)).astype(np.int32)
        ctx.lhs.importRegularAndQuantize(cuda(X), cuda(thr))
        A = (X[None] > thr[:, :, None]).sum(0).astype(np.int16)
        check()
        bit = int(A[7, 11]) >> 5 & 1
        (ctx.lhs.unset if bit else ctx.lhs.set)(5, 7, 11)
        A[7, 11] ^= 32
        check()
    finally:
        deallocGEMMContext(ctx)
