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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("bw", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("planes,length,maxlen", [(1, 1, 1), (1, 129, 129), (3, 85, 90), (1, 257, 300)])
def test_fp32_register_tiles(D, bw, planes, length, maxlen):
    """Sums of D products in fp32: the kernel's chain and the oracle's differ by at most
    2 D 2^-24 of the sum of the products' magnitudes, which is at most |y| |Pi column| = |y|
    <= sqrt(D) times the largest centroid (Pi is orthogonal)."""
    tq = _get_quantizer(bw, D, DEV, 42)
    codes, norms = _rows(planes, maxlen, D, bw, 7)
    N = planes * length
    for dtype in (torch.float32, torch.bfloat16):
        guard = torch.full((N + 64, D), -12352.0, dtype=dtype, device=DEV)
        out = guard[32:32 + N].view(planes, length, D)
        dequantize_rows(codes.to(DEV)[:, :length], norms.to(DEV)[:, :length], tq.centroids, tq.Pi, bw, D, out=out,
                        mode="exact")
        o = orc.OracleQuantizer.get(bw, D, 42)
        ref = orc.dequantize_rows(codes[:, :length].contiguous(), norms[:, :length].contiguous(), o.centroids, o.Pi,
                                  bw, D)
        bound = 2 * D * 2.0 ** -24 * D ** 0.5 * float(o.centroids.abs().max()) * norms[:, :length, None].float()
        if dtype == torch.bfloat16:
            bound = bound + ref.abs() * 2.0 ** -8
        assert ((out.float().cpu() - ref.reshape(out.shape)).abs() <= bound).all()
        assert (guard[:32] == -12352.0).all() and (guard[32 + N:] == -12352.0).all()
