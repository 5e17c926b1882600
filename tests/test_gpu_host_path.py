"""The native host path at its limits: what it passes on to the general path, and the
errors it raises itself."""
import pytest
import torch

import cases
from helpers import assert_attention_close, oracle_case, to_device
from oracle import tq_oracle as orc
from winnow_b200 import _lib, packed_attention as pa
from winnow_b200.cache import _get_quantizer
from winnow_b200.engine_step import DecodeSession
from winnow_b200.packed_attention_cuda import packed_decode_attention
from winnow_b200.page_pool import PagePool

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


def _session(dtype=torch.float16, B=3, Hq=8, Hkv=2, D=128):
    tq = _get_quantizer(4, D, DEV, 42)
    pool = PagePool(num_layers=1, num_pages=12, num_kv_heads=Hkv, page_size=16, nb_k=64, nb_v=64, device=DEV)
    owners = [f"r{b}" for b in range(B)]
    pool.ensure_many(owners, [20] * B)
    s = DecodeSession(pool, owners, [0] * B, k_quant=tq, v_quant=tq, head_dim=D, q_heads=Hq, dtype=dtype, max_tokens=32)
    s.begin_step()
    return s, pool


def _step_inputs(seed, B=3, Hq=8, Hkv=2, D=128):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn(B, h, 1, D, generator=g).half().to(DEV) for h in (Hkv, Hkv, Hq)]


def _unaligned(x):
    flat = torch.empty(x.numel() + 3, dtype=x.dtype, device=DEV)[3:]
    return flat.view(x.shape).copy_(x)


def _strided(x):
    wide = torch.empty(*x.shape[:-1], 2 * x.shape[-1], dtype=x.dtype, device=DEV)[..., ::2]
    return wide.copy_(x)


@pytest.mark.parametrize("change", [_unaligned, _strided, lambda x: x.float(), lambda x: x.cpu(),
                                    lambda x: x.transpose(0, 1).contiguous().transpose(0, 1),
                                    lambda x: x.clone().requires_grad_()],
                         ids=["unaligned", "strided", "other type", "on the host", "transposed", "with a gradient"])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_staging_takes_what_copy_takes(change, which):
    """K, V or the query in a form the one-launch copy does not serve: the step is the same."""
    s, pool = _session()
    x = _step_inputs(which)
    s.k_in.zero_(), s.v_in.zero_(), s.q_in.zero_()
    want = s.layer(0, *x).clone()
    pages = [t.clone() for t in (pool.k_pages, pool.k_norms, pool.v_pages, pool.v_norms)]
    for t in (pool.k_pages, pool.v_pages):
        t.zero_()
    s.k_in.zero_(), s.v_in.zero_(), s.q_in.zero_()
    x[which] = change(x[which])
    with torch.no_grad():
        got = s.layer(0, *x)
    assert torch.equal(got, want)
    assert all(torch.equal(a, b) for a, b in zip(pages, (pool.k_pages, pool.k_norms, pool.v_pages, pool.v_norms)))
    s.check()


def test_staging_refuses_a_shape_that_does_not_fit():
    s, _ = _session()
    k, v, q = _step_inputs(7)
    with pytest.raises(RuntimeError):
        s.layer(0, k[:2], v, q)
    assert torch.equal(s.layer(0, k, v[:1].expand_as(v), q), s.layer(0, k, v[:1], q))        # (broadcast, as copy_ does)


def test_decode_passes_on_what_it_does_not_serve():
    """A wider status word, a result with its own strides, a query that is not contiguous."""
    c = C("pass", 52, 2, 8, 2, 128, (40, 9), 16, 4, 4)
    q, okv, _ = oracle_case(c)
    kv, scale = to_device(okv, DEV), orc.default_scale(128)
    ref = orc.tiled_attention(q, okv, scale)
    status = torch.zeros(1, dtype=torch.int64, device=DEV)
    assert_attention_close(packed_decode_attention(q.to(DEV), kv, scale, check_page_ids=False, status=status), ref)
    assert int(status) == 0
    kv.page_table[0, 1] = 10 ** 6
    packed_decode_attention(q.to(DEV), kv, scale, check_page_ids=False, status=status)
    assert int(status) == _lib.STATUS_BAD_PAGE
    kv.page_table[0, 1] = okv.page_table[0, 1].item()
    pinned = torch.zeros(1, dtype=torch.int32).pin_memory()
    assert_attention_close(packed_decode_attention(q.to(DEV), kv, scale, check_page_ids=False, status=pinned), ref)
    into = torch.empty(2, 16, 1, 128, device=DEV)[:, ::2]
    got = packed_decode_attention(_strided(q.to(DEV)), kv, scale, check_page_ids=False, out=into)
    assert got is into
    assert_attention_close(into, ref)
    for bad in (dict(out=into.half()), dict(out=into[:1]), dict(out=torch.empty(2, 8, 1, 128))):
        with pytest.raises(pa.UnsupportedLayout):
            packed_decode_attention(q.to(DEV), kv, scale, check_page_ids=False, **bad)
    kv.k_norms = kv.k_norms.float()
    with pytest.raises(pa.UnsupportedLayout):
        packed_decode_attention(q.to(DEV), kv, scale, check_page_ids=False)
