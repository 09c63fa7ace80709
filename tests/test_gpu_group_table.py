"""Job tables of grouped imports: more operands than a launch carries in its parameters (24), so every import writes the
group's device table anew, beside groups small enough to need none.  Imports of new tensors on alternating streams, an
import recorded into the caller's own graph between plain ones, and the group's captured graph, which keeps a table of
its own.  Every import's results are kept and compared."""
import numpy as np
import pytest

from gemmbitserial_gb300 import _capi, datagen
from gemmbitserial_gb300.api import allocGEMMContext, deallocGEMMContext
from gemmbitserial_gb300.grouped import Group

pytestmark = pytest.mark.gpu
# direct (rows of 16 bytes) and staged operands, popcount and tensor-core problems
DIMS = [(4, 256, 70), (40, 363, 90), (200, 1024, 130), (8, 64, 33), (1, 512, 300), (129, 160, 129), (16, 999, 61),
        (33, 48, 200)]


@pytest.fixture(scope="module", autouse=True)
def lib(gbs_lib):
    import torch
    assert torch.cuda.is_available()
    return gbs_lib


class Problems:
    def __init__(self, count):
        self.dims = [DIMS[i % len(DIMS)] for i in range(count)]
        self.ctxs = [allocGEMMContext(M, K, N, 2, 2, False, True) for M, K, N in self.dims]
        self.grp = Group(self.ctxs)
        self.sets = [self.operands(datagen.SEED_BASE + 1400 + 100 * i) for i in range(3)]

    def operands(self, seed):
        """(lhs tensors, rhs tensors, expected results) of every problem."""
        import torch
        ops = [(datagen.operand(seed + 2 * i, M, K, 2, "u"), datagen.operand(seed + 2 * i + 1, N, K, 2, "s"))
               for i, (M, K, N) in enumerate(self.dims)]
        return ([torch.from_numpy(a).cuda() for a, _ in ops], [torch.from_numpy(b).cuda() for _, b in ops],
                [(b.astype(np.int64) @ a.astype(np.int64).T).astype(np.int32) for a, b in ops])

    def results(self, stream):
        """Copies of every result, taken on the stream."""
        import torch
        out = []
        for c, (M, _, N) in zip(self.ctxs, self.dims):
            out.append(torch.empty(N, M, dtype=torch.int32, device="cuda"))
            _capi.check(_capi.load().gbs_get_result(c._h, out[-1].data_ptr(), stream.cuda_stream))
        return out

    def check(self, kept):
        import torch
        torch.cuda.synchronize()
        for i, (got, which) in enumerate(kept):
            for t, w in zip(got, self.sets[which][2]):
                assert np.array_equal(t.cpu().numpy(), w), (i, which)

    def run(self, which, stream):
        """One import and GEMM of set `which` with a copy of its results, all on the stream."""
        self.grp.import_(self.sets[which][0], self.sets[which][1], stream=stream)
        self.grp.gemm(stream=stream)
        return self.results(stream), which


@pytest.fixture(params=[4, 16])
def problems(request):
    p = Problems(request.param)
    yield p
    p.grp.free()
    for c in p.ctxs:
        deallocGEMMContext(c)


def test_imports_on_two_streams(problems):
    import torch
    streams, kept = (torch.cuda.Stream(), torch.cuda.Stream()), []
    torch.cuda.synchronize()
    for r in range(9):  # ordered by the caller, with no host synchronisation
        s = streams[r % 2]
        s.wait_stream(streams[1 - r % 2])
        kept.append(problems.run(r % 3, s))
    problems.check(kept)
    assert problems.grp.status() == _capi.GBS_OK


@pytest.mark.parametrize("before", [0, 1])
def test_import_recorded_between_plain_ones(problems, before):
    import torch
    s, kept = torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for _ in range(before):
        kept.append(problems.run(0, s))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):  # the recorded table is allocated meanwhile
        problems.grp.import_(problems.sets[1][0], problems.sets[1][1], stream=s)
        problems.grp.gemm(stream=s)
    for r in range(3):
        kept.append(problems.run(2 * (r % 2), s))
        with torch.cuda.stream(s):
            graph.replay()
        kept.append((problems.results(s), 1))
    problems.check(kept)
    assert problems.grp.status() == _capi.GBS_OK


def test_captured_graph_keeps_its_table(problems):
    import torch
    s1, s2, kept = torch.cuda.Stream(), torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for which, s, other in ((0, s1, s2), (2, s2, s1)):
        problems.grp.capture(problems.sets[which][0], problems.sets[which][1], stream=s)
        for _ in range(2):
            other.wait_stream(s)
            kept.append(problems.run(1, other))
            s.wait_stream(other)
            problems.grp.replay(stream=s)  # packs the tensors it was captured with
            kept.append((problems.results(s), which))
    problems.check(kept)
    assert problems.grp.status() == _capi.GBS_OK
