"""Calls that decode in fp32 throughout (queries, centroids, probabilities and value
weights are 32-bit floats), against 64-bit arithmetic: head_dim 64 whatever the size of the
values, head_dim 128 with layouts the tensor-core scan does not take."""
import math

import pytest
import torch

import cases
from helpers import oracle_case, to_device
from oracle import tq_oracle as orc
from winnow_b200.packed_attention_cuda import decode_workspace, packed_decode_attention
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
    check(got, ref, size, top, 64, 251)


def check(got, ref, size, top, D, keys):
    # u = 2^-24.  A score sums D products twice (rotation, then centroids) and takes three more
    # roundings: off by at most (2 D + 3) u |q| |k|; a probability by that times ln 2 and by 2^-22
    # for exp2, its quotient by twice as much.  The value sum takes a rounding per key of a chain
    # (`keys`: a warp's share of 3001, or all), some 20 to merge and D to rotate back.
    u = 2.0 ** -24
    bound = 2 * ((2 * D + 3) * u * math.log(2) * top + 2.0 ** -22) + (keys + 20 + D) * u
    err = (got[:, :, 0].double() - ref).norm(dim=-1)
    assert (err <= bound * size).all(), float((err / size.clamp_min(1e-300)).max() / bound)


def test_layouts_the_tensor_core_scan_does_not_take():
    """Pages 2^31 bytes apart, and a workspace off its alignment."""
    c = C("far", 43, 2, 8, 2, 128, (1, 40), 16, 4, 4, 0.02)
    q, okv, _ = oracle_case(c)
    kv, scale = to_device(okv, "cuda"), orc.default_scale(128)
    ref, size, top = exact(q.cuda(), kv, scale)
    for splits in (None, 2):
        ws = decode_workspace(2, 8, 2, 128, kv.page_table.shape[1], 16, splits or 0, "cuda")
        off = torch.zeros(ws.numel() + 16, dtype=torch.uint8, device="cuda")[4:]
        got = packed_decode_attention(q.cuda(), kv, scale, num_splits=splits, workspace=off)
        check(got, ref, size, top, 128, 40)
    P, H, S, NB = kv.k_pages.shape
    far = torch.zeros((P - 1 << 31) + H * S * NB, dtype=torch.uint8, device="cuda")
    far = far.as_strided((P, H, S, NB), (1 << 31, S * NB, NB, 1))
    far.copy_(kv.k_pages)
    kv.k_pages = far
    for splits in (None, 2):
        check(packed_decode_attention(q.cuda(), kv, scale, num_splits=splits), ref, size, top, 128, 40)
