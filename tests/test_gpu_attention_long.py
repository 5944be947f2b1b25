"""Attention beyond one KV tile: rows whose scores grow from tile to tile (the accumulator is then
rescaled), the one- and two-query-tile forms of a work item, ragged ends of both, items without a
valid key between others, against the CPU oracle."""
import numpy as np
import pytest

from util import assert_close_f16, to_dev

pytestmark = pytest.mark.gpu


def _run(hom, cuda, qkv, lens, heads):
    import torch

    bs, seq, width = qkv.shape
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    out = torch.full((bs, seq, width // 3), float("nan"), dtype=torch.float16, device=cuda)
    hom.nvteBertAttentionF16(to_dev(qkv, cuda), to_dev(cu, cuda), out, 0.125, heads)
    hom.synchronize()
    return out.cpu().numpy(), cu


@pytest.mark.parametrize("order", ["rising", "falling", "some rows"])
@pytest.mark.parametrize("bs,seq,heads,lens", [(2, 512, 2, [512, 300]), (40, 384, 3, None)])
def test_scores_that_grow_from_tile_to_tile(hom, cuda, oracle, order, bs, seq, heads, lens):
    """Scores of about 20 per KV tile step (2^29 in the exponentials): every row's reference has to
    follow (rising), must not (falling), or follows in some rows of a warp only."""
    rng = np.random.default_rng(5)
    lens = np.array(lens) if lens is not None else rng.integers(1, seq + 1, bs)
    qkv = rng.normal(0, 0.3, (bs, seq, 3, heads, 64)).astype(np.float32)
    tile = np.arange(seq) // 128
    level = tile if order != "falling" else tile.max() - tile
    qkv[:, :, 0, :, 0] = 8.0  # one dimension carries the level of a key to every query
    if order == "some rows":
        qkv[:, ::3, 0, :, 0] = 0.0
    qkv[:, :, 1, :, 0] = (20.0 * level)[None, :, None]
    qkv = qkv.reshape(bs, seq, 3 * heads * 64).astype(np.float16)
    got, cu = _run(hom, cuda, qkv, lens, heads)
    assert_close_f16(got, oracle.attention_f16(qkv, cu, heads, 0.125), f"{order} {bs}x{seq}")


@pytest.mark.parametrize("bs,seq,heads,lens", [
    (1, 129, 1, [129]),             # one tile per item; a second tile of one row
    (3, 130, 2, [0, 130, 1]),       # nothing valid, everything, one key
    (2, 255, 30, [255, 128]),       # 120 tiles: one each
    (3, 257, 30, [257, 256, 129]),  # two tiles per item, the last group with a single row
    (70, 200, 3, None),             # more items than CTAs, ragged
    (5, 640, 12, [0, 640, 5, 513, 0]),
])
def test_work_item_forms(hom, cuda, oracle, bs, seq, heads, lens):
    rng = np.random.default_rng(seq)
    lens = np.array(lens) if lens is not None else rng.integers(0, seq + 1, bs)
    qkv = rng.normal(0, 1, (bs, seq, 3 * heads * 64)).astype(np.float16)
    got, cu = _run(hom, cuda, qkv, lens, heads)
    assert_close_f16(got, oracle.attention_f16(qkv, cu, heads, 0.125), f"{bs}x{seq}x{heads}")


def test_a_row_with_nan_scores_stays_a_zero_row(hom, cuda):
    """A NaN in a query makes the row's sum NaN; such rows are written as zeros and no other row
    changes."""
    rng = np.random.default_rng(7)
    qkv = rng.normal(0, 1, (1, 300, 3 * 64)).astype(np.float16)
    clean, _ = _run(hom, cuda, qkv, np.array([300]), 1)
    bad = qkv.copy()
    bad[0, [3, 140, 299], :64] = np.nan
    got, _ = _run(hom, cuda, bad, np.array([300]), 1)
    rest = np.setdiff1d(np.arange(300), [3, 140, 299])
    assert np.array_equal(got[0, rest].view(np.uint16), clean[0, rest].view(np.uint16))
    assert (got[0, [3, 140, 299]] == 0).all()
