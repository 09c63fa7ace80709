"""Column-major threshold imports at the edges of their 32 x 32 pieces: single rows and columns, tall and flat sources,
remainders, every element type, no thresholds and more than a byte counts, unsorted and infinite thresholds, NaN and
infinite elements; the planes by export and the digits by a GEMM on the tensor cores.  Exact against the definition:
the index of the first threshold with x <= threshold, its low bits."""
import ctypes as C

import numpy as np
import pytest

from gemmbitserial_gb300 import _capi
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial

pytestmark = pytest.mark.gpu
SHAPES = [(1, 1), (1, 5000), (5000, 1), (31, 33), (32, 32), (33, 31), (65, 257), (40001, 3), (3, 40001), (257, 640)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


def codes(src, thr):
    """src [rows][cols], thr [nthres][rows]"""
    if not len(thr):
        return src.astype(np.int64) & 0xFF
    out = np.zeros(src.shape, np.int64)
    searching = np.ones(src.shape, bool)
    for t in thr:
        searching &= ~(src <= t[:, None])
        out += searching
    return out & 0xFF


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("dtype", [np.int8, np.uint8, np.int16, np.int32, np.float32])
@pytest.mark.parametrize("nthres,bits", [(0, 3), (1, 1), (3, 2), (7, 3), (15, 4), (260, 8)])
def test_codes(shape, dtype, nthres, bits):
    import torch
    M, K = shape
    N = 40
    rng = np.random.default_rng(2000 + nthres + M)
    lo, hi = (0, 50) if dtype == np.uint8 else (-25, 25)
    src = rng.integers(lo, hi, (M, K)).astype(dtype)
    thr = rng.integers(lo, hi, (nthres, M)).astype(dtype)
    if nthres and nthres != 3:
        thr.sort(axis=0)  # 3: unsorted
    if dtype == np.float32 and nthres:
        src[rng.random(src.shape) < 0.05] = np.nan
        src[rng.random(src.shape) < 0.05] = np.inf
        src[rng.random(src.shape) < 0.05] = -np.inf
        if nthres > 3:
            thr[-1, ::3] = np.inf
            thr[0, ::4] = -np.inf
    want = codes(src, thr) & ((1 << bits) - 1)
    ctx = allocGEMMContext(M, K, N, bits, 2, False, False)
    try:
        if bits <= 4:
            ctx.set_pipe(_capi.GBS_PIPE_TC)
        ctx.lhs.importRegularAndQuantize(torch.from_numpy(np.ascontiguousarray(src.T)).cuda(),
                                         torch.from_numpy(thr).cuda() if nthres else None, nthres, readColMajor=True)
        got = np.zeros((M, K), np.int32)
        _capi.check(_capi.load().gbs_export(ctx._h, 0, C.c_void_p(got.ctypes.data), None))
        assert np.array_equal(got, want)
        B = rng.integers(0, 4, (N, K)).astype(np.int8)
        ctx.rhs.importRegular(torch.from_numpy(B).cuda())
        gemmBitSerial(ctx)
        assert np.array_equal(ctx.res.reshape(N, M), (B.astype(np.float64) @ want.T.astype(np.float64)).astype(np.int32))
    finally:
        deallocGEMMContext(ctx)
