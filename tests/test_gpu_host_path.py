"""The native host path at its limits: what it passes on to the general path, and the
errors it raises itself."""
import pytest
import torch

import cases
from helpers import oracle_case, to_device
from oracle import tq_oracle as orc
from winnow_b200.packed_attention_cuda import packed_decode_attention

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
C = cases.AttnCase


def test_no_memory_for_the_workspace():
    """torch.OutOfMemoryError, as torch's own allocations raise it."""
    c = C("oom", 51, 2, 8, 2, 128, (40, 9), 16, 4, 4)
    q, okv, _ = oracle_case(c)
    kv, B = to_device(okv, DEV), 64
    kv.page_table = kv.page_table.new_full((B, 8192), -1)             # 131072 tokens: 1024 splits of 64 x 8 rows
    kv.seq_lens = kv.seq_lens.new_zeros(B)
    q = q.to(DEV).repeat(B // 2, 1, 1, 1)
    packed_decode_attention(q[:, :, :, :], kv, 1.0, check_page_ids=False)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(DEV).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            packed_decode_attention(q, kv, 1.0, num_splits=1024, check_page_ids=False)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert not packed_decode_attention(q, kv, 1.0, num_splits=1024, check_page_ids=False).any()
