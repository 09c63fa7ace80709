"""SM-pair tiles with K split over independent pairs (the built-in rule for few tiles and a long K): every split, row
and column remainders, stages that do not divide, repeated and concurrent launches.  Bit-exact against int64."""
import ctypes as C

import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu

# (M, K, N, split the rule takes: 0 for whatever it is)
CASES = [(256, 9216, 4096, 4), (300, 16384, 270, 8), (1000, 16000, 1000, 4), (257, 10007, 2049, 4), (1500, 12000, 1280, 2),
         (2048, 8192, 256, 8), (256, 16384, 256, 8), (511, 1500, 300, 0)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


def make(M, K, N, wa, ea, wb, eb, seed):
    import torch
    A = datagen.operand(datagen.SEED_BASE + seed, M, K, wa, ea)
    B = datagen.operand(datagen.SEED_BASE + seed + 1, N, K, wb, eb)
    ctx = allocGEMMContext(M, K, N, wa, wb, ea != "u", eb != "u")
    ctx.set_pipe(_capi.GBS_PIPE_TC)
    ctx.lhs.importRegular(torch.from_numpy(A).cuda())
    ctx.rhs.importRegular(torch.from_numpy(B).cuda())
    return ctx, (B.astype(np.float64) @ A.astype(np.float64).T).astype(np.int64).astype(np.int32)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[:3])))
@pytest.mark.parametrize("enc", [(3, "u", 2, "s"), (1, "b", 4, "s")])
def test_splits(case, enc):
    M, K, N, want_splits = case
    ctx, want = make(M, K, N, *enc, seed=1001)
    try:
        for _ in range(3):
            gemmBitSerial(ctx)
            assert np.array_equal(ctx.res.reshape(N, M), want)
        bn, sp, kind = C.c_int(), C.c_int(), C.c_int()
        _capi.check(_capi.load().gbs_debug_last_pair(ctx._h, C.byref(bn), C.byref(sp), C.byref(kind)))
        if want_splits:
            assert (bn.value, sp.value, kind.value) == (256, want_splits, 0)
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(ctx)


def test_two_streams_at_once():
    """Split GEMMs of two contexts in flight together: no pair waits for another, so any interleaving finishes."""
    import torch
    a, want_a = make(512, 16384, 768, 2, "u", 2, "s", seed=1011)
    b, want_b = make(256, 16384, 1024, 1, "b", 3, "u", seed=1021)
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    try:
        for _ in range(20):
            gemmBitSerial(a, stream=s1)
            gemmBitSerial(b, stream=s2)
        torch.cuda.synchronize()
        assert np.array_equal(a.res.reshape(want_a.shape), want_a)
        assert np.array_equal(b.res.reshape(want_b.shape), want_b)
        assert _capi.load().gbs_debug_tc_error() == 0
    finally:
        deallocGEMMContext(a)
        deallocGEMMContext(b)
