"""What the append and the contiguous cache refuse before anything is launched, on tensors
without storage: a kernel given these arguments would read outside its buffers."""
from types import SimpleNamespace

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from winnow_b200 import _lib, packed_attention as pa, packed_backend as pb
from winnow_b200.cache import TQPackedLayer
from winnow_b200.packed_attention_cuda import DecodePlan


@pytest.fixture
def fake():
    with FakeTensorMode():
        yield


def _append_args(B=4, rows=4, lens=4, device="cuda", Pi_device="cuda"):
    D, H, n, S, P = 128, 2, 8, 16, 5
    x = [torch.empty(B, H, n, D, dtype=torch.float16, device=device) for _ in range(2)]
    pages = [torch.empty(P, H, S, 64, dtype=torch.uint8, device=device) for _ in range(2)]
    norms = [torch.empty(P, H, S, dtype=torch.float16, device=device) for _ in range(2)]
    tq = SimpleNamespace(Pi=torch.empty(D, D, device=Pi_device), centroids=torch.empty(16, device=Pi_device),
                         boundaries=torch.empty(15, device=Pi_device), bit_width=4)
    return [*x, pages[0], norms[0], pages[1], norms[1], torch.empty(rows, 1, dtype=torch.int32, device=device),
            torch.empty(lens, dtype=torch.int32, device=device), tq, tq]


@pytest.mark.parametrize("rows,lens", [(3, 4), (4, 3), (1, 1)])
def test_append_needs_a_table_row_and_a_length_per_sequence(fake, rows, lens):
    with pytest.raises(ValueError, match="row for each of 4"):
        pb.AppendPlan(*_append_args(rows=rows, lens=lens))


def test_append_needs_its_quantizers_on_the_device(fake):
    with pytest.raises(_lib.BackendError):
        pb.AppendPlan(*_append_args(Pi_device="cpu"))


@pytest.mark.parametrize("which", ["workspace", "status"])
def test_buffers_in_pageable_host_memory(fake, which):
    args = _append_args()
    on_host = torch.empty(1 << 20, dtype=torch.uint8 if which == "workspace" else torch.int32, device="cpu")
    quant = pa.Quantizer.from_tq(args[8])
    kv = pa.PackedKV(*args[2:8], quant, quant, 128)
    with pytest.raises(_lib.BackendError, match=which):
        DecodePlan(torch.empty(4, 8, 1, 128, device="cuda"), kv, 1.0, check_page_ids=False, **{which: on_host})
    if which == "status":
        with pytest.raises(_lib.BackendError, match=which):
            pb.AppendPlan(*args, status=on_host)


@pytest.mark.parametrize("k_shape,v_shape", [((3, 2, 8, 128), None), ((1, 2, 8, 128), None), ((8, 2, 8, 128), None),
                                             ((4, 1, 8, 128), None), ((4, 2, 8, 128), (4, 2, 1, 128)),
                                             ((4, 2, 8, 128), (1, 2, 8, 128))])
def test_contiguous_cache_appends_only_its_own_shape(fake, monkeypatch, k_shape, v_shape):
    """Other shapes go part by part, where assignment broadcasts them or raises."""
    called = []
    monkeypatch.setattr(pb, "append_tokens", lambda *a, **k: called.append(1))
    layer = TQPackedLayer.__new__(TQPackedLayer)
    layer._out_dim, layer._shape, layer._tq = 0, (4, 2, 128), None
    layer._ring_len = torch.zeros(4, dtype=torch.int32, device="cuda")
    layer._ring_table = layer._k = layer._v = (None, None)
    ks = torch.empty(k_shape, dtype=torch.float16, device="cuda")
    vs = torch.empty(v_shape or k_shape, dtype=torch.float16, device="cuda")
    assert not layer._store_both(ks, vs, 0, 8) and not called
    own = torch.empty(4, 2, 8, 128, dtype=torch.float16, device="cuda")
    assert layer._store_both(own, own, 0, 8) and called


_NO_STORAGE = """
import sys
sys.path[:0] = {path!r}
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from test_refusals import _append_args
from winnow_b200 import _lib, packed_attention as pa, packed_backend as pb
host = _lib.host()
with FakeTensorMode():
    args = _append_args()
    k, v, kp, kn, vp, vn, table, lens, tq, _ = args
    q = torch.empty(4, 8, 1, 128, dtype=torch.float16, device="cuda")
    quant = pa.Quantizer.from_tq(tq)
    kv = pa.PackedKV(kp, kn, vp, vn, table, lens, quant, quant, 128)
    status = torch.empty(1, dtype=torch.int32, device="cuda")
    for call in (lambda: pb.append_tokens(*args), lambda: host.append(*args, -1, status),
                 lambda: host.stage(k, k, v, v, q, q), lambda: host.decode(q, kv, 1.0, 0, None, None, status),
                 lambda: host.decode(q, kv, 1.0, 4, torch.empty_like(q), None, None),
                 lambda: host.attend(q, kv, 1.0, None)):
        try:
            call()
        except Exception as e:
            print("raised", type(e).__name__)
"""


def test_tensors_without_storage_raise():
    """In a process of its own: a C++ exception that leaves the interpreter's C function ends it."""
    import subprocess
    import sys
    code = _NO_STORAGE.format(path=[p for p in sys.path if p])
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert done.stdout.count("raised ") == 6, done.stdout
