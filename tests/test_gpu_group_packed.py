"""Packed plans of a group's tensor-core problems: every width and encoding of the larger side, as 4-bit floats where
they allow it, written by the grouped import and by the expansion of planes that single imports left, at the tiles'
edges; and the popcount kernels' matrix-vector outputs."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext, gemmBitSerial
from gemmbitserial_gb300.grouped import Group

pytestmark = pytest.mark.gpu
DIMS = [(17, 1, 19), (127, 129, 128), (129, 383, 128), (300, 130, 257), (16, 1025, 513)]  # rows, K, rows
KINDS = [(b, e) for b in (1, 2, 3, 4) for e in ("u", "s")]  # 1-bit "s" is bipolar


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


@pytest.mark.parametrize("bits,enc", KINDS)
@pytest.mark.parametrize("expanded", [False, True])
def test_packed_plan(bits, enc, expanded, monkeypatch):
    import torch
    monkeypatch.setenv("GBS_GROUP_PIPE", "tc")
    monkeypatch.setenv("GBS_TCG_NIBBLES", "1")
    rng = np.random.default_rng(77 + 10 * bits + (enc == "s"))
    ops, ctxs = [], []
    for M, K, N in DIMS:
        wb = int(rng.integers(1, 5))
        a = datagen.operand(int(rng.integers(1 << 30)), M, K, bits, "b" if (bits, enc) == (1, "s") else enc)
        b = datagen.operand(int(rng.integers(1 << 30)), N, K, wb, "u")
        if M < N:  # either side may be the larger, packed, one
            ops.append((b, a))
            ctxs.append(allocGEMMContext(N, K, M, wb, bits, False, enc == "s"))
        else:
            ops.append((a, b))
            ctxs.append(allocGEMMContext(M, K, N, bits, wb, enc == "s", False))
    g = Group(ctxs)
    try:
        assert g.stats()["tc_kernel"] == "nibbles"
        dev = [(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()) for a, b in ops]
        if expanded:
            for c, (a, b) in zip(ctxs, dev):
                c.lhs.importRegular(a)
                c.rhs.importRegular(b)
        else:
            g.import_([a for a, _ in dev], [b for _, b in dev])
        g.gemm()
        torch.cuda.synchronize()
        assert g.status() == _capi.GBS_OK
        for c, (a, b) in zip(ctxs, ops):
            want = b.astype(np.int64) @ a.astype(np.int64).T
            assert np.array_equal(c.res.reshape(want.shape), want)
    finally:
        g.free()
        for c in ctxs:
            deallocGEMMContext(c)


@pytest.mark.parametrize("bits", [(1, 1), (2, 2), (1, 2), (3, 1)])
@pytest.mark.parametrize("K", [1, 255, 8192, 12288, 12289, 24600])
def test_matrix_vector(bits, K):
    """Steps of two words a lane at their edges, in the grouped kernel and the single one."""
    import torch
    wa, wb = bits
    rng = np.random.default_rng(K)
    dims, ops, ctxs = [(1, 1), (37, 1), (3, 2)], [], []
    for M, N in dims:
        ops.append((rng.integers(0, 1 << wa, (M, K)).astype(np.int8), rng.integers(0, 1 << wb, (N, K)).astype(np.int8)))
        ctxs.append(allocGEMMContext(M, K, N, wa, wb, False, False))
    g = Group(ctxs)
    try:
        dev = [(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()) for a, b in ops]
        g.import_([a for a, _ in dev], [b for _, b in dev])
        g.gemm()
        torch.cuda.synchronize()
        assert g.status() == _capi.GBS_OK
        for c, (a, b) in zip(ctxs, ops):
            want = b.astype(np.int64) @ a.astype(np.int64).T
            assert np.array_equal(c.res.reshape(want.shape), want)
            c.set_pipe(_capi.GBS_PIPE_POPC)
            gemmBitSerial(c)
            assert np.array_equal(c.res.reshape(want.shape), want)
    finally:
        g.free()
        for c in ctxs:
            deallocGEMMContext(c)
