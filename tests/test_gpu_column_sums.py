"""LayerNorm-on-A GEMM: the column sums of B it needs, for shapes at the edges of the column-sum
kernel (fewer columns than a block, a column tail, fewer and more rows than its warps), for weights
that are declared (sums kept), not declared (computed on every call) and seen first under capture."""
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
