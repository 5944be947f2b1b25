"""LayerNorm-on-A GEMM: the column sums of B it needs, for shapes at the edges of the column-sum
kernel (fewer columns than a block, a column tail, fewer and more rows than its warps), for weights
that are declared (sums kept), not declared (computed on every call) and seen first under capture."""
import time

import numpy as np
import pytest

from util import assert_close_f16, to_dev

pytestmark = pytest.mark.gpu


def _case(m, n, k, seed):
    rng = np.random.default_rng(seed)
    A = rng.normal(0, 1, (1, m, k)).astype(np.float16)
    B = rng.normal(0.02, 0.05, (1, k, n)).astype(np.float16)  # a mean, so that wrong sums show
    rstd = rng.uniform(0.5, 2.0, m).astype(np.float16)
    shift = rng.normal(0, 1, m).astype(np.float16)
    a, b = A[0].astype(np.float64), B[0].astype(np.float64)
    want = rstd.astype(np.float64)[:, None] * (a @ b) + shift.astype(np.float64)[:, None] * b.sum(0)[None, :]
    return A, B, rstd, shift, want[None].astype(np.float16)


@pytest.mark.parametrize("declared", [False, True])
@pytest.mark.parametrize("m,n,k", [(5, 8, 8), (64, 72, 40), (130, 200, 264), (128, 3072, 768)])
def test_column_sums(hom, cuda, m, n, k, declared):
    import torch

    A, B, rstd, shift, want = _case(m, n, k, m + n)
    tA, tB, tV, tM = (to_dev(x, cuda) for x in (A, B, rstd, shift))
    tD = torch.zeros((1, m, n), dtype=torch.float16, device=cuda)
    if declared:
        hom.declare_weights(tB)
    try:
        for _ in range(2):
            tD.zero_()
            hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
            hom.synchronize()
            assert_close_f16(tD.cpu().numpy(), want, f"{m}x{n}x{k}")
        tB.mul_(-1)  # new contents: a renewed declaration drops what was derived from the old ones
        if declared:
            hom.declare_weights(tB)
        hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
        hom.synchronize()
        assert_close_f16(tD.cpu().numpy(), -want, "negated weights")
    finally:
        if declared:
            hom.forget_weights(tB)


def test_column_sums_of_a_weight_first_seen_under_capture(hom, cuda):
    import torch

    A, B, rstd, shift, want = _case(64, 256, 128, 3)
    tA, tB, tV, tM = (to_dev(x, cuda) for x in (A, B, rstd, shift))
    tD = torch.zeros((1, 64, 256), dtype=torch.float16, device=cuda)
    hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)  # library set-up outside the capture
    hom.synchronize()
    hom.declare_weights(tB)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    try:
        hom.set_stream(stream.cuda_stream)
        with torch.cuda.graph(graph, stream=stream):
            hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
        tD.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert_close_f16(tD.cpu().numpy(), want, "replayed")
    finally:
        hom.use_torch_stream()
        hom.forget_weights(tB)


def _partials(x):
    """{sum, sum of squares} of every row per 64-column group, [groups, rows, 2] fp32."""
    g = x.astype(np.float32).reshape(x.shape[0], -1, 64)
    return np.ascontiguousarray(np.stack([g.sum(-1), (g * g).sum(-1)], axis=-1).transpose(1, 0, 2))


@pytest.mark.parametrize("first", ["kn", "nk"])
def test_a_square_weight_read_in_both_layouts(hom, cuda, first):
    """One declared buffer taken as [K, N] by one entry point and as [N, K] by another: each gets the
    sums of its own layout, whichever of them came first."""
    import torch

    m, n = 64, 128
    A, B, rstd, shift, want_kn = _case(m, n, n, 7)
    a, b = A[0].astype(np.float64), B[0].astype(np.float64)
    mean, var = a.mean(-1, keepdims=True), a.var(-1, keepdims=True)
    want_nk = (((a - mean) / np.sqrt(var + 1e-12)) @ b.T)[None]
    tA, tB, tV, tM, tS = (to_dev(x, cuda) for x in (A, B, rstd, shift, _partials(A[0])))
    tD = torch.zeros((1, m, n), dtype=torch.float16, device=cuda)

    def kn():
        hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
        hom.synchronize()
        assert_close_f16(tD.cpu().numpy(), want_kn, "[K, N]")

    def nk():
        hom.homGemmDeferredLayernormF16(tA, tS, tB, None, None, tD, None, weights_nk=True)
        hom.synchronize()
        assert_close_f16(tD.cpu().numpy(), want_nk, "[N, K]")

    hom.declare_weights(tB)
    try:
        for call in (kn, nk, kn) if first == "kn" else (nk, kn, nk):
            call()
    finally:
        hom.forget_weights(tB)


def test_a_captured_call_follows_a_rewritten_weight(hom, cuda):
    """A graph captured when the weight's sums were already kept: rewriting the weight and declaring
    it again (which gives the kept sums back) leaves the graph valid, and it follows the contents."""
    import torch

    A, B, rstd, shift, want = _case(64, 256, 128, 11)
    tA, tB, tV, tM = (to_dev(x, cuda) for x in (A, B, rstd, shift))
    tD = torch.zeros((1, 64, 256), dtype=torch.float16, device=cuda)
    hom.declare_weights(tB)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    try:
        hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
        hom.synchronize()
        hom.set_stream(stream.cuda_stream)
        with torch.cuda.graph(graph, stream=stream):
            hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
        for factor in (1, -1, 0.5):
            tB.copy_(torch.from_numpy(B)).mul_(factor)
            hom.declare_weights(tB)
            tD.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert_close_f16(tD.cpu().numpy(), want.astype(np.float64) * factor, f"weights x {factor}")
    finally:
        hom.use_torch_stream()
        hom.forget_weights(tB)


def test_captured_calls_do_not_share_their_sums(hom, cuda):
    """Two graphs captured on one stream, with different weights, replayed on two streams at once;
    then both destroyed and captured again, their memory being given back in the meantime (by the
    declaration inside the next capture, or before)."""
    import torch

    cases = [_case(256, 512, 512, seed) for seed in (21, 22)]
    other = torch.zeros(64, dtype=torch.float16, device=cuda)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    dev = [[to_dev(x, cuda) for x in c[:4]] + [torch.zeros((1, 256, 512), dtype=torch.float16, device=cuda)]
           for c in cases]
    torch.cuda.synchronize()
    try:
        hom.set_stream(streams[0].cuda_stream)
        for _ in range(3):
            graphs = [torch.cuda.CUDAGraph() for _ in cases]
            for graph, (tA, tB, tV, tM, tD) in zip(graphs, dev):
                with torch.cuda.graph(graph, stream=streams[0]):
                    hom.declare_weights(other)
                    hom.forget_weights(other)
                    for _ in range(8):
                        hom.cutlassLayernormGemmF16(tA, tB, None, tD, tV, tM)
            for _ in range(20):
                for graph, stream in zip(graphs, streams):
                    with torch.cuda.stream(stream):
                        graph.replay()
            torch.cuda.synchronize()
            for case, d in zip(cases, dev):
                assert_close_f16(d[4].cpu().numpy(), case[4], "replayed on two streams")
                d[4].zero_()
            del graph, graphs
            time.sleep(0.2)  # CUDA reports the end of a graph from a thread of its own
    finally:
        hom.use_torch_stream()


def test_a_graph_keeps_what_was_derived_from_its_weights(hom, cuda):
    """What a graph was captured with (kept column sums, the re-pitched copy of an odd-N weight) stays
    until the graph is gone, although the weights have been declared again in between."""
    import torch

    m, k, n = 64, 2048, 8196  # the copy of the second weight: 33.6 MB
    A, B, _, _, _ = _case(m, 256, k, 31)
    a, b = A[0].astype(np.float64), B[0].astype(np.float64)
    mean, var = a.mean(-1, keepdims=True), a.var(-1, keepdims=True)
    want = (((a - mean) / np.sqrt(var + 1e-12)) @ b)[None]
    V = np.random.default_rng(32).normal(0, 0.02, (1, k, n)).astype(np.float16)
    rows = torch.from_numpy(A).to(cuda)
    tS, tB, tV = (to_dev(x, cuda) for x in (_partials(A[0]), B, V))
    tD = torch.zeros((1, m, 256), dtype=torch.float16, device=cuda)
    tL = torch.zeros((1, m, n), dtype=torch.float16, device=cuda)
    want_l = a @ V[0].astype(np.float64)

    def call():
        hom.homGemmDeferredLayernormF16(rows, tS, tB, None, None, tD, None)
        hom.cutlassGemmF16(rows, tV, None, tL)

    def free_memory():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    for t in (tB, tV):
        hom.declare_weights(t)
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    try:
        call()
        hom.synchronize()
        hom.set_stream(stream.cuda_stream)
        with torch.cuda.graph(graph, stream=stream):
            call()
        before = free_memory()
        for t in (tB, tV):
            hom.declare_weights(t)
        assert free_memory() - before < 16 << 20, "the copy that the graph reads was freed"
        tD.zero_()
        tL.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert_close_f16(tD.cpu().numpy(), want, "kept sums")
        assert_close_f16(tL.cpu().numpy()[0], want_l, "re-pitched copy")
        before = free_memory()
        del graph
        for _ in range(100):  # CUDA reports the end of a graph from a thread of its own
            hom.declare_weights(tV)
            if free_memory() - before >= 32 << 20:
                break
            time.sleep(0.05)
        assert free_memory() - before >= 32 << 20, "the copy outlived the graph"
    finally:
        hom.use_torch_stream()
        for t in (tB, tV):
            hom.forget_weights(t)


def test_calls_on_two_streams_do_not_share_their_sums(hom, cuda):
    """Weights that are not declared, one per stream, calls on the two streams interleaved."""
    import torch

    cases = [_case(64, 2048, 2048, seed) for seed in (41, 42)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    dev = [[to_dev(x, cuda) for x in c[:4]] + [torch.zeros((1, 64, 2048), dtype=torch.float16, device=cuda)
                                               for _ in range(40)] for c in cases]

    def call(i):
        for stream, d in zip(streams, dev):
            hom.set_stream(stream.cuda_stream)
            hom.cutlassLayernormGemmF16(d[0], d[1], None, d[4 + i], d[2], d[3])

    try:
        call(0)
        torch.cuda.synchronize()
        gate = torch.cuda.Event()
        torch.cuda._sleep(50_000_000)  # both queues fill behind this, then run at the same time
        gate.record()
        for stream in streams:
            stream.wait_event(gate)
        for i in range(40):
            call(i)
        torch.cuda.synchronize()
    finally:
        hom.use_torch_stream()
    for case, d in zip(cases, dev):
        assert_close_f16(d[4].cpu().numpy(), case[4], "first call")
        for tD in d[5:]:
            assert torch.equal(tD, d[4])


@pytest.mark.parametrize("declared", [False, True])
def test_a_first_call_beside_a_capture(hom, cuda, declared):
    """The first call for a declared weight, or on a new stream, allocates (and waits); it may do so
    while the same thread captures another stream (torch's default capture mode), and leaves that
    capture valid."""
    import torch

    cases = [_case(64, 256, 128, seed) for seed in (51, 52)]
    (A, B, V, M, D), (A2, B2, V2, M2, D2) = [
        [to_dev(x, cuda) for x in c[:4]] + [torch.zeros((1, 64, 256), dtype=torch.float16, device=cuda)]
        for c in cases]
    captured, beside = torch.cuda.Stream(), torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    if declared:
        hom.declare_weights(B2)
    try:
        with torch.cuda.graph(graph, stream=captured):
            hom.set_stream(captured.cuda_stream)
            hom.cutlassLayernormGemmF16(A, B, None, D, V, M)
            hom.set_stream(beside.cuda_stream)
            hom.cutlassLayernormGemmF16(A2, B2, None, D2, V2, M2)
            hom.set_stream(captured.cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        assert_close_f16(D.cpu().numpy(), cases[0][4], "captured")
        assert_close_f16(D2.cpu().numpy(), cases[1][4], "beside the capture")
    finally:
        hom.use_torch_stream()
        if declared:
            hom.forget_weights(B2)
