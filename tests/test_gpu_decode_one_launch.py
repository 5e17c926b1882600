"""The one-launch decode kernel at its edges: windows and warps that a length
leaves empty or part-filled, every cluster size, both head dimensions, all width
pairs, group sizes 1..8, page sizes 16..64, against the CPU oracle at the
operator's tolerance (max-abs 2e-3, relative L2 1e-3)."""
import pytest
import torch

import cases
from helpers import assert_attention_close, oracle_case, to_device
from oracle import tq_oracle as orc
from winnow_b200 import _lib
from winnow_b200.packed_attention_cuda import packed_decode_attention

pytestmark = pytest.mark.gpu
C = cases.AttnCase

SHAPES = [
    # empty, one token, around a tile, a window, and the last warp's share
    C("edges_d128", 1, 8, 4, 1, 128, (0, 1, 15, 16, 17, 31, 32, 33), 16, 4, 4),
    C("edges_d64", 2, 8, 7, 1, 64, (0, 1, 15, 16, 17, 31, 32, 33), 16, 4, 4),
    # one block per group (more than 74 groups), ragged
    C("cluster1", 3, 19, 16, 4, 128, tuple(range(3, 3 + 19 * 37, 37)), 32, 8, 8),
    # clusters of 2, 4 and 8 blocks whose last warps are empty for the short sequences
    C("cluster2", 4, 20, 6, 3, 128, (513, 1) + (40,) * 18, 16, 4, 6),
    C("cluster4", 5, 5, 32, 4, 128, (1025, 3, 900, 32, 770), 64, 6, 6),
    C("cluster8", 6, 2, 16, 2, 128, (2049, 64), 16, 4, 4),
    C("cluster8_d64", 7, 2, 10, 2, 64, (2050, 100), 32, 6, 6),
    C("d64_mixed", 8, 3, 8, 8, 64, (700, 33, 16), 16, 4, 6),
    C("d64_8bit", 9, 3, 6, 1, 64, (300, 95, 1), 16, 8, 8),
    # large logits: windows scored again in fp32
    C("huge_d64", 10, 2, 14, 2, 64, (90, 600), 16, 4, 4, 40.0),
    C("huge_d128", 11, 2, 28, 4, 128, (90, 600), 16, 6, 6, 40.0),
    # more groups than multiprocessors
    C("many_groups_d64", 12, 80, 4, 2, 64, tuple(1 + (i * 29) % 131 for i in range(80)), 16, 4, 4),
]


@pytest.mark.parametrize("c", SHAPES, ids=lambda c: c.name)
def test_one_launch_matches_the_oracle(c):
    q, okv, _ = oracle_case(c)
    ref = orc.tiled_attention(q, okv, orc.default_scale(c.D))
    kv = to_device(okv, "cuda")
    packed_decode_attention(q.cuda(), kv, orc.default_scale(c.D))
    before = _lib.lib().wtq_launch_count()
    got = packed_decode_attention(q.cuda(), kv, orc.default_scale(c.D))
    assert _lib.lib().wtq_launch_count() - before == 1
    assert_attention_close(got, ref)


def test_refused_pages_and_positions_are_reported():
    c = C("bad", 20, 2, 8, 2, 128, (100, 80), 16, 4, 4)
    q, okv, _ = oracle_case(c)
    kv = to_device(okv, "cuda")
    kv.page_table = kv.page_table.clone()
    kv.page_table[0, 2] = kv.k_pages.shape[0] + 7          # outside the pool
    kv.seq_lens = kv.seq_lens.clone()
    kv.seq_lens[1] = kv.page_table.shape[1] * c.S + 5      # beyond the table
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    out = packed_decode_attention(q.cuda(), kv, orc.default_scale(c.D), check_page_ids=False, status=status)
    assert int(status.item()) == _lib.STATUS_BAD_PAGE | _lib.STATUS_BAD_POSITION
    assert torch.isfinite(out).all()


@pytest.mark.parametrize("B,Hq,Hkv,widths,width_tokens,launches", [
    (18, 32, 8, (4, 4), 131072, 3), (16, 32, 8, (4, 4), 8192, 3), (16, 32, 8, (4, 4), 2048, 1),
    (32, 28, 4, (8, 8), 1984, 1), (32, 28, 4, (8, 8), 4096, 3), (16, 32, 8, (6, 6), 2048, 3), (16, 32, 8, (4, 6), 4096, 3),
    (4, 32, 8, (4, 4), 65536, 3), (8, 32, 8, (4, 4), 8192, 3), (1, 32, 8, (4, 4), 16384, 1), (1, 32, 8, (4, 4), 131072, 3)])
def test_long_tables_go_to_the_whole_chip(B, Hq, Hkv, widths, width_tokens, launches):
    """One launch lasts as long as the longest sequence may be: tables that admit one which
    the split-K path would share out go there, with the same result either way."""
    c = C("width", 60, B, Hq, Hkv, 128, (300,) + (40,) * (B - 1), 16, *widths)
    q, okv, _ = oracle_case(c)
    kv = to_device(okv, "cuda")
    wide = torch.full((B, width_tokens // 16), -1, dtype=torch.int32, device="cuda")
    wide[:, :kv.page_table.shape[1]] = kv.page_table
    kv.page_table = wide
    q, scale = q.cuda(), orc.default_scale(128)
    packed_decode_attention(q, kv, scale, check_page_ids=False)
    before = _lib.lib().wtq_launch_count()
    got = packed_decode_attention(q, kv, scale, check_page_ids=False)
    assert _lib.lib().wtq_launch_count() - before == launches
    assert_attention_close(got, packed_decode_attention(q, kv, scale, num_splits=2, check_page_ids=False))
