"""head_dim 64 decodes in fp32 whatever the size of the values: queries, centroids,
probabilities and value weights are 32-bit floats, against 64-bit arithmetic."""
import math

import pytest
import torch

import cases
from helpers import oracle_case, to_device
from oracle import tq_oracle as orc
from winnow_b200.packed_attention_cuda import packed_decode_attention
from winnow_b200.packing import unpack

pytestmark = pytest.mark.gpu
C = cases.AttnCase


def exact(q, kv, scale):
    """(result in fp64, sum of p |v| of every row, largest |q| |k| in log2 units)."""
    B, Hq, _, D = q.shape
    out, top = torch.zeros(B, Hq, D, dtype=torch.float64, device=q.device), 0.0
    size = torch.zeros(B, Hq, dtype=torch.float64, device=q.device)
    for b in range(B):
        L = int(kv.seq_lens[b])
        if not L:
            continue
        ids = kv.page_table[b, :-(-L // kv.page_size)].long()
        sides = []
        for pages, norms, quant in ((kv.k_pages, kv.k_norms, kv.k_quant), (kv.v_pages, kv.v_norms, kv.v_quant)):
            idx = unpack(pages[ids].contiguous(), quant.bit_width, D).long()
            y = (quant.centroids.double()[idx] @ quant.Pi.double()) * norms[ids].double()[..., None]
            y = y.permute(1, 0, 2, 3).reshape(pages.shape[1], -1, D)[:, :L]
            sides.append(y.repeat_interleave(Hq // pages.shape[1], 0))
        k, v = sides
        s = torch.einsum("hd,hld->hl", q[b, :, 0].double(), k) * scale
        out[b] = torch.einsum("hl,hld->hd", s.softmax(-1), v)
        size[b] = (s.softmax(-1) * v.norm(dim=-1)).sum(-1)
        top = max(top, float((q[b, :, 0].double().norm(dim=-1)[:, None] * k.norm(dim=-1)).max()) * scale / math.log(2))
    return out, size, top


@pytest.mark.parametrize("widths", [(4, 4), (4, 6), (6, 6), (8, 8)])
@pytest.mark.parametrize("heads", [(1, 1), (4, 1), (14, 2), (16, 2)])
@pytest.mark.parametrize("v_scale,q_scale", [(1.0, 1.0), (1e-4, 1.0), (1e-6, 1.0), (1.0, 8.0)])
def test_fp32_against_64_bits(widths, heads, v_scale, q_scale):
    c = C("d64", 41, 5, heads[0], heads[1], 64, (0, 1, 33, 500, 3001), 16, *widths, q_scale)
    q, okv, _ = oracle_case(c)
    kv, scale = to_device(okv, "cuda"), orc.default_scale(64)
    kv.v_norms = (kv.v_norms.float() * v_scale).half()
    ref, size, top = exact(q.cuda(), kv, scale)
    got = packed_decode_attention(q.cuda(), kv, scale)
    assert got.dtype == torch.float32
    # u = 2^-24.  A score sums 64 products twice (rotation, then centroids) and takes three more
    # roundings: off by at most 131 u |q| |k|; a probability by that times ln 2 and by 2^-22 for
    # exp2, its quotient by twice as much.  The value sum of 3001 keys takes a rounding per key of
    # a warp's share (at most 251), some 20 to merge and 64 to rotate back.
    u = 2.0 ** -24
    bound = 2 * (131 * u * math.log(2) * top + 2.0 ** -22) + (251 + 20 + 64) * u
    err = (got[:, :, 0].double() - ref).norm(dim=-1)
    assert (err <= bound * size).all(), float((err / size.clamp_min(1e-300)).max() / bound)
