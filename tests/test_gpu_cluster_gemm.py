"""The GEMM form that cuts K over a thread-block cluster (tile rows 1 and 2 with a split of 2..8):
edges of tiles, uneven shares of rows and of K blocks, both weight layouts, every epilogue operand,
against the CPU oracle; and the rule that picks it."""
import numpy as np
import pytest

from util import assert_bits_equal, assert_close_f16, to_dev


def _run(hom, cuda, A, B, C, *, row, split, act=0, alpha=1.0, beta=0.0, nk=False, alias=False):
    import torch

    tA, tB = to_dev(A, cuda), to_dev(B, cuda)
    tC = None if C is None else to_dev(C, cuda)
    tD = tC if alias else torch.full((1, A.shape[1], B.shape[1] if nk else B.shape[2]), 7.0, dtype=torch.float16,
                                     device=cuda)
    if nk:  # this entry point has no split argument: the automatic choice
        hom.nvteGemmF16(tA, tB, tC if beta else tD, tD, activation=act, alpha=alpha, beta=beta)
    else:
        hom.cutlassGemmF16(tA, tB, tC if beta else tD, tD, activation=act, alpha=alpha, beta=beta, gemmNum=row,
                           splitKFactor=split)
    hom.synchronize()
    return tD.cpu().numpy()


def _operands(m, n, k, seed):
    rng = np.random.default_rng(seed)
    return (rng.normal(0, 1, (1, m, k)).astype(np.float16), rng.normal(0, 0.05, (1, k, n)).astype(np.float16),
            rng.normal(0, 1, (1, m, n)).astype(np.float16))


@pytest.mark.gpu
@pytest.mark.parametrize("row", [1, 2])
@pytest.mark.parametrize("m,n,k,split", [
    (1, 8, 128, 2),        # one row, one 8-column piece, one K block per CTA
    (7, 72, 136, 3),       # fewer rows than columns of a piece; a ragged last K block
    (63, 768, 768, 8),     # rows do not divide by the parts
    (65, 200, 520, 5),     # a column tail that is no multiple of 64
    (128, 768, 3072, 7),   # a full tile, 7 x 19 receive rows (the largest receive buffer)
    (129, 136, 264, 4),    # a second row block with a single row: most owners have none
    (385, 1024, 1024, 6),  # more clusters than run at once
    (257, 64, 512, 8),
])
def test_cluster_split_matches_the_oracle(hom, cuda, oracle, row, m, n, k, split):
    A, B, C = _operands(m, n, k, 1000 + m + split)
    got = _run(hom, cuda, A, B, C, row=row, split=split, beta=1.0, alias=True)
    assert_close_f16(got, oracle.gemm_f16(A, B, C, beta=1.0), "residual in place")
    again = _run(hom, cuda, A, B, C, row=row, split=split, beta=1.0, alias=True)
    assert_bits_equal(again, got, "the parts are added in a fixed order")
    bias = C[:, :1, :].copy()
    got = _run(hom, cuda, A, B, bias, row=row, split=split, alpha=0.5, beta=2.0, act=1)
    assert_close_f16(got, oracle.gemm_f16(A, B, bias, alpha=0.5, beta=2.0, act=1), "scaled, bias row, GELU")


@pytest.mark.gpu
@pytest.mark.parametrize("row,m,n,k,split", [
    (1, 1024, 1152, 256, 2),  # 144 tiles: clusters, the second wave partly filled
    (1, 1024, 1208, 256, 2),  # 152 tiles: serial split on persistent CTAs
    (2, 1281, 1400, 264, 4),  # 121 tiles, clusters
    (2, 1409, 1480, 264, 4),  # 144 tiles, serial
    (1, 300, 200, 136, 16),   # more parts than K blocks: three, as clusters
])
def test_asked_for_splits_on_both_sides_of_the_rule(hom, cuda, oracle, row, m, n, k, split):
    A, B, C = _operands(m, n, k, 3000 + m + split)
    got = _run(hom, cuda, A, B, C, row=row, split=split, beta=1.0)
    assert_close_f16(got, oracle.gemm_f16(A, B, C, beta=1.0), "residual")


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k", [(16, 768, 768), (64, 2304, 768), (77, 768, 3072), (200, 1024, 4096)])
def test_automatic_choice_with_weights_stored_nk(hom, cuda, oracle, m, n, k):
    assert hom.gemm_query_tile(m, n, k, 0)["split_k"] >= 2
    A, B, C = _operands(m, n, k, 2000 + m)
    got = _run(hom, cuda, A, np.ascontiguousarray(B.transpose(0, 2, 1)), C, row=0, split=1, beta=1.0, nk=True)
    assert_close_f16(got, oracle.gemm_f16(A, B, C, beta=1.0), "[1, N, K] weights")


@pytest.mark.gpu
@pytest.mark.parametrize("nk", [False, True])
@pytest.mark.parametrize("m,n,k,split", [(64, 1024, 4096, 8), (200, 136, 3072, 2), (128, 768, 3072, 5)])
def test_declared_weights_with_a_share_longer_than_the_ring(hom, cuda, oracle, m, n, k, split, nk, tmp_path):
    """The first K blocks of a declared weight are requested before the kernel that writes A has
    finished, the others as the ring (six stages, four with 128 columns) comes round."""
    import torch

    A, B, C = _operands(m, n, k, 4000 + m)
    want = oracle.gemm_f16(A, B, C, beta=1.0)
    tB = to_dev(np.ascontiguousarray(B.transpose(0, 2, 1)) if nk else B, cuda)
    half, tC = to_dev(A / 2, cuda), to_dev(C, cuda)
    tA = torch.zeros((1, m, k), dtype=torch.float16, device=cuda)
    tD = torch.zeros((1, m, n), dtype=torch.float16, device=cuda)
    table = tmp_path / "tuned.txt"
    hom.declare_weights(tB)
    try:
        for row, stages in ((1, 6), (2, 4)):
            assert -(-k // 64) // split > stages
            table.write_text(f"{m} {n} {k} 0 {row} {split}\n")  # the [N, K] entry takes its split from here
            assert hom.gemm_tune_load(table) == 1
            for _ in range(3):
                tA.zero_()
                hom.elementwise("Add", "F16", half, half, tA)
                if nk:
                    hom.nvteGemmF16(tA, tB, tC, tD, beta=1.0)
                else:
                    hom.cutlassGemmF16(tA, tB, tC, tD, beta=1.0)
                hom.synchronize()
                assert_close_f16(tD.cpu().numpy(), want, f"row {row}")
    finally:
        hom.forget_weights(tB)


def test_the_rule_splits_only_where_all_clusters_run_at_once(hom):
    """Rows 1 and 2, at most eight parts, no more parts than K blocks, no more CTAs than SMs; no
    split at all where N is not a multiple of 8 or the output has more tiles than the chip."""
    for m in (1, 64, 100, 128, 300, 512, 1000, 4096, 30000):
        for n, k in ((768, 768), (2304, 768), (3072, 768), (768, 3072), (1024, 4096), (64, 64), (30520, 768)):
            q = hom.gemm_query_tile(m, n, k, 0)
            if q["split_k"] > 1:
                tiles = -(-m // 128) * -(-n // q["bn"])
                assert q["row"] in (1, 2) and q["split_k"] <= min(8, -(-k // 64))
                assert tiles * q["split_k"] <= 148
    assert hom.gemm_query_tile(64, 770, 3072, 0)["split_k"] == 1
    assert hom.gemm_query_tile(4096, 768, 3072, 0)["split_k"] == 1
