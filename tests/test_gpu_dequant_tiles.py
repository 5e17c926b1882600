"""Dequantisation at the edges of its tiles: the call over two tensors against two
calls, and the fp32 register-tiled kernel against the oracle."""
import ctypes

import pytest
import torch

from oracle import tq_oracle as orc
from winnow_b200 import _lib
from winnow_b200.cache import _get_quantizer, dequantize_rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _rows(planes, maxlen, D, bw, seed):
    g = torch.Generator().manual_seed(seed)
    codes = torch.randint(0, 256, (planes, maxlen, D * bw // 8), generator=g, dtype=torch.uint8)
    return codes, (torch.rand(planes, maxlen, generator=g) * 50 + 0.5).half()


@pytest.mark.parametrize("planes,length,maxlen", [(1, 1, 1), (3, 41, 64), (2, 64, 64), (1, 129, 140), (8, 2400, 2401)])
@pytest.mark.parametrize("bw,dtype,D", [(4, torch.bfloat16, 128), (6, torch.float16, 128), (8, torch.bfloat16, 128),
                                        (4, torch.float32, 128), (3, torch.float16, 128), (4, torch.bfloat16, 64)])
def test_two_tensors_are_two_calls(planes, length, maxlen, bw, dtype, D):
    """Bit for bit, with the rows of both outputs guarded on either side."""
    tq = _get_quantizer(bw, D, DEV, 42)
    sides = [[t.to(DEV) for t in _rows(planes, maxlen, D, bw, s)] for s in (1, 2)]
    N = planes * length
    guards = [torch.full((N + 64, D), -12352.0, dtype=dtype, device=DEV) for _ in range(2)]
    outs = [x[32:32 + N] for x in guards]
    pair = ctypes.c_void_p * 2
    _lib.check(_lib.lib().wtq_dequant_pair(
        pair(*(s[0].data_ptr() for s in sides)), pair(*(s[1].data_ptr() for s in sides)), tq.centroids.data_ptr(),
        tq.Pi.data_ptr(), pair(*(o.data_ptr() for o in outs)), _lib.dtype_code(dtype), bw, D, N, length, maxlen,
        _lib.stream_ptr(torch.device(DEV))))
    for (codes, norms), guard, out in zip(sides, guards, outs):
        one = torch.empty(planes, length, D, dtype=dtype, device=DEV)
        dequantize_rows(codes[:, :length], norms[:, :length], tq.centroids, tq.Pi, bw, D, out=one)
        assert torch.equal(out, one.view(N, D))
        assert (guard[:32] == -12352.0).all() and (guard[32 + N:] == -12352.0).all()
