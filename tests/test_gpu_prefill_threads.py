"""Chunked prefill from several threads on one stream: every call has a workspace of its own."""
import threading

import pytest
import torch

import cases
from helpers import oracle_case, to_device
from oracle import tq_oracle as orc
from winnow_b200.packed_attention_cuda import packed_prefill_attention

pytestmark = pytest.mark.gpu


def test_threads_that_share_a_stream():
    """Far enough ahead of the device that launches wait for room in its queue: there the
    launches of one call and another's interleave."""
    calls = []
    for i, lens in enumerate(((3000, 800), (700, 2900), (2500, 2500))):
        _, okv, _ = oracle_case(cases.AttnCase(f"thread{i}", 71 + i, 2, 8, 2, 128, lens, 16, 4, 4))
        q = torch.randn(2, 8, 24, 128, generator=torch.Generator().manual_seed(i)).cuda() / 11.0
        calls.append((q, to_device(okv, "cuda")))
    scale = orc.default_scale(128)
    want = [packed_prefill_attention(q, kv, scale, check_page_ids=False).clone() for q, kv in calls]
    torch.cuda.synchronize()
    got, start = [[] for _ in calls], threading.Barrier(len(calls))

    def work(i):
        q, kv = calls[i]
        start.wait()
        for _ in range(600):
            got[i].append(packed_prefill_attention(q, kv, scale, check_page_ids=False))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [sum(not torch.equal(x, want[i]) for x in outs) for i, outs in enumerate(got)] == [0] * len(calls)
