"""Chunked prefill where a few keys carry a row: the rounding of their probabilities to
16 bits cancels between the value sum and its denominator."""
import math

import pytest
import torch

from winnow_b200 import packed_attention as pa
from winnow_b200.cache import _get_quantizer
from winnow_b200.packed_attention_cuda import packed_prefill_attention
from winnow_b200.packing import unpack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("widths", [(4, 4), (4, 6), (6, 6), (8, 8)])
@pytest.mark.parametrize("lead", [5.1, 5.3, 5.55, 6.8, 7.4])
def test_two_keys_carry_the_rows(widths, lead):
    D, S, H, Q, L, first, second = 128, 16, 2, 16, 208, 3, 130
    g = torch.Generator().manual_seed(int(10 * lead))
    kq, vq = _get_quantizer(widths[0], D, DEV, 42), _get_quantizer(widths[1], D, DEV, 43)
    pages = [torch.randint(0, 256, (L // S, H, S, D * w // 8), generator=g, dtype=torch.uint8) for w in widths]
    norms = [torch.rand(L // S, H, S, generator=g) * 0.5 + 2.0, torch.rand(L // S, H, S, generator=g) * 4 + 8.0]
    # the second key: the codes of the first, longer; scores of about 60 and 60 + lead, all others far below
    pages[0][second // S, :, second % S] = pages[0][first // S, :, first % S]
    norms[0][first // S, :, first % S] = 11.0
    norms[0][second // S, :, second % S] = 11.0 * (60 + lead) / 60
    pages, norms = [p.to(DEV) for p in pages], [n.half().to(DEV) for n in norms]
    kv = pa.PackedKV(pages[0], norms[0], pages[1], norms[1],
                     torch.arange(L // S, dtype=torch.int32, device=DEV)[None],
                     torch.tensor([L], dtype=torch.int32, device=DEV), pa.Quantizer.from_tq(kq),
                     pa.Quantizer.from_tq(vq), D)
    scale = D ** -0.5

    def rows(side, tq, w):                               # (H, L, D) codes, (H, L) norms
        idx = unpack(pages[side], w, D).long().permute(1, 0, 2, 3).reshape(H, L, D)
        return idx, norms[side].permute(1, 0, 2).reshape(H, L)

    idx, n = rows(0, kq, widths[0])
    k = (kq.centroids.double()[idx] @ kq.Pi.double()) * n[..., None].double()
    q = k[:, first] * (60 * math.log(2) / scale) / k[:, first].square().sum(-1, keepdim=True)
    q = q.repeat_interleave(4, 0)[None, :, None].expand(1, 4 * H, Q, D).float().contiguous()
    s = torch.einsum("hd,hld->hl", q[0, :, 0].double(), k.repeat_interleave(4, 0)) * scale
    idx, n = rows(1, vq, widths[1])
    v = ((vq.centroids.half()[idx] * n[..., None]).double() @ vq.Pi.double()).repeat_interleave(4, 0)   # operands as rounded
    ref = torch.einsum("hl,hld->hd", s.softmax(-1), v)
    got = packed_prefill_attention(q, kv, scale)[0].double()
    # A probability is off by at most 2^-11 of itself.  With it in both sums the weights move by
    # 2 w (1 - w) 2^-11 of |v|, w <= 2^-lead the smaller weight; scores in fp32 move them by
    # another ln 2 x 65 x 128 x 2^-24 x w, and 1e-5 is left for fp32 sums and split operands.
    w = 2.0 ** -lead
    bound = 2 * w * 2.0 ** -11 + w * math.log(2) * 65 * 128 * 2.0 ** -24 + 1e-5
    err = (got - ref[:, None]).norm(dim=-1) / v.norm(dim=-1).amax(-1)[:, None]
    assert (err <= bound).all(), float(err.max() / bound)
