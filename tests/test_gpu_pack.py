"""The pack kernels over every source form: element types, row lengths around the
vector widths, sources that start off alignment, row- and column-major, plain
and threshold imports, alone and grouped.  The planes (padding included) are
compared bit for bit with codes computed by numpy, and the tensor-core operands an
import writes through the GEMM that reads them."""
import numpy as np
import pytest

from gemmbitserial_gb300 import datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial
from gemmbitserial_gb300.grouped import Group

pytestmark = pytest.mark.gpu

DTYPES = {"int8": np.int8, "uint8": np.uint8, "int16": np.int16, "int32": np.int32, "float32": np.float32}
# row lengths: below, at and above a 4-element group, a 32-column chunk and a 1024-column unit
SHAPES = [(1, 1), (3, 31), (5, 32), (2, 48), (67, 33), (64, 100), (9, 363), (130, 257), (33, 1024), (17, 1056),
          (31, 2051), (259, 64), (40, 2048), (5, 1028), (6, 1100), (24, 3072)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


def codes(x, bits, signed):
    """The stored code of every element (importRegular<T>, integer-valued input)."""
    if bits == 1 and signed and x.dtype != np.uint8:
        return (x > 0).astype(np.int64)
    return x.astype(np.int64) & ((1 << bits) - 1)


def check_planes(planes, want, bits):
    rows, cols = want.shape
    nb, rows_a, wpr = planes.shape
    assert nb == bits
    got = np.unpackbits(planes.view(np.uint8).reshape(nb, rows_a, wpr * 8), axis=2, bitorder="little")
    full = np.zeros((nb, rows_a, wpr * 64), np.uint8)
    for b in range(nb):
        full[b, :rows, :cols] = (want >> b) & 1
    assert np.array_equal(got, full)


def on_device(x, col_major, offset):
    """x in the order the import reads it, `offset` elements past an aligned address."""
    import torch
    flat = np.ascontiguousarray(x.T if col_major else x).reshape(-1)
    buf = torch.zeros(flat.size + offset, dtype=torch.from_numpy(flat).dtype, device="cuda")
    buf[offset:] = torch.from_numpy(flat).cuda()
    return buf[offset:]


@pytest.mark.parametrize("col_major", [False, True], ids=["row", "col"])
@pytest.mark.parametrize("dtype", list(DTYPES))
def test_planes_of_every_source(dtype, col_major):
    rng = np.random.default_rng(11)
    for n, (rows, cols) in enumerate(SHAPES):
        for bits, signed in [(1, False), (1, True), (3, False), (4, True), (8, False)]:
            lo, hi = (-(1 << (bits - 1)), (1 << (bits - 1)) - 1) if signed and bits > 1 else (0, (1 << bits) - 1)
            if bits == 1 and signed:
                x = rng.integers(0, 2, (rows, cols)) * 2 - 1
            else:
                x = rng.integers(lo, hi + 1, (rows, cols))
            x = x.astype(DTYPES[dtype])
            ctx = allocGEMMContext(rows, cols, 2, bits, 1, signed, False)
            try:
                ctx.lhs.importRegular(on_device(x, col_major, (0, 1, 3, 16)[n % 4]), readColMajor=col_major)
                check_planes(ctx.lhs.planes(), codes(x, bits, signed), bits)
            finally:
                deallocGEMMContext(ctx)


@pytest.mark.parametrize("col_major", [False, True], ids=["row", "col"])
@pytest.mark.parametrize("dtype", list(DTYPES))
def test_threshold_planes(dtype, col_major):
    import torch
    rng = np.random.default_rng(12)
    for n, (rows, cols) in enumerate(SHAPES):
        for bits, nthres in [(1, 1), (3, 7), (2, 9), (8, 200)]:
            x = rng.integers(0 if dtype == "uint8" else -100, 120, (rows, cols)).astype(DTYPES[dtype])
            t = rng.integers(0 if dtype == "uint8" else -100, 120, (nthres, rows)).astype(DTYPES[dtype])
            if n % 2:  # unsorted ones give the first crossing
                t = np.sort(t, axis=0)
            below = x[None] <= t[:, :, None]
            want = np.where(below.any(0), below.argmax(0), nthres) & ((1 << bits) - 1)
            ctx = allocGEMMContext(rows, cols, 2, bits, 1, False, False)
            try:
                ctx.lhs.importRegularAndQuantize(on_device(x, col_major, (0, 1, 3, 16)[n % 4]),
                                                 torch.from_numpy(t).cuda(), nthres, readColMajor=col_major)
                check_planes(ctx.lhs.planes(), want, bits)
            finally:
                deallocGEMMContext(ctx)


def test_float_values_past_the_integers():
    """The low byte of a truncation to 64 bits: saturated, infinite, NaN and fractional inputs, and thresholds that
    a NaN never crosses."""
    import torch
    x = np.array([[0.9, -0.9, 255.0, 256.0, 300.7, 2147483520.0, 2147483648.0, 4e18, 9.3e18, 1e30, np.inf, np.nan,
                   -np.inf, -1e30, -3e9, -1.0, -129.5, 7.999]], np.float32)
    low = [0, 0, 255, 0, 44, 128, 0, 0, 255, 255, 255, 0, 0, 0, 0, 255, 127, 7]
    low[7] = int(np.int64(np.float32(4e18))) & 255
    ctx = allocGEMMContext(1, x.shape[1], 2, 8, 1, False, False)
    try:
        ctx.lhs.importRegular(torch.from_numpy(x).cuda())
        check_planes(ctx.lhs.planes(), np.array([low]), 8)
        t = np.array([[-1.0], [0.0], [255.0]], np.float32)
        ctx.lhs.importRegularAndQuantize(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda(), 3)
        below = x[None] <= t[:, :, None]
        check_planes(ctx.lhs.planes(), np.where(below.any(0), below.argmax(0), 3), 8)
    finally:
        deallocGEMMContext(ctx)


@pytest.mark.parametrize("shape", [(256, 300, 272), (70, 777, 520), (300, 1030, 33)])
@pytest.mark.parametrize("enc", [(4, "s", 2, "u"), (1, "b", 3, "s"), (3, "u", 1, "b")])
def test_column_major_imports_write_the_tensor_core_operands(shape, enc):
    """The GEMM after column-major imports, against int64 products."""
    import torch
    M, K, N = shape
    wa, ea, wb, eb = enc
    A = datagen.operand(datagen.SEED_BASE + 301, M, K, wa, ea)
    B = datagen.operand(datagen.SEED_BASE + 302, N, K, wb, eb)
    ctx = allocGEMMContext(M, K, N, wa, wb, ea != "u", eb != "u")
    try:
        for _ in range(2):
            ctx.lhs.importRegular(torch.from_numpy(np.ascontiguousarray(A.T)).cuda(), readColMajor=True)
            ctx.rhs.importRegular(torch.from_numpy(np.ascontiguousarray(B.T)).cuda(), readColMajor=True)
            gemmBitSerial(ctx)
            assert np.array_equal(ctx.res.reshape(N, M), (B.astype(np.int64) @ A.astype(np.int64).T).astype(np.int32))
            A, B = np.ascontiguousarray(A[::-1]), np.ascontiguousarray(B[::-1])
    finally:
        deallocGEMMContext(ctx)


def test_grouped_import_of_mixed_sources():
    """Direct (aligned 1-byte) and staged (wide, unaligned) operands in one group: planes of every operand."""
    import torch
    rng = np.random.default_rng(13)
    dims = [(1, 64, 70), (9, 363, 40), (130, 257, 33), (33, 1024, 300), (64, 48, 257), (7, 8192, 65), (256, 2304, 169)]
    kinds = ["int8", "int16", "int32", "uint8", "int8", "int8", "int32"]
    ops, ctxs = [], []
    for (M, K, N), kind in zip(dims, kinds):
        ops.append([rng.integers(0, 4, (r, K)).astype(DTYPES[k]) for r, k in ((M, kind), (N, "int8"))])
        ctxs.append(allocGEMMContext(M, K, N, 2, 2, False, False))
    try:
        g = Group(ctxs)
        try:
            g.import_([torch.from_numpy(a).cuda() for a, _ in ops], [torch.from_numpy(b).cuda() for _, b in ops])
            g.gemm()
            for c, (a, b) in zip(ctxs, ops):
                check_planes(c.lhs.planes(), a.astype(np.int64), 2)
                check_planes(c.rhs.planes(), b.astype(np.int64), 2)
                want = (b.astype(np.int64) @ a.astype(np.int64).T).astype(np.int32)
                assert np.array_equal(c.res.reshape(want.shape), want)
        finally:
            g.free()
    finally:
        for c in ctxs:
            deallocGEMMContext(c)
