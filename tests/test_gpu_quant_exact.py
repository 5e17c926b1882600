"""The tensor-core quantiser returns the bytes of the sequential fp32 chains: all
widths, source types and strides, vector counts around its passes of 16 and 64
vectors, and vectors built to put coordinates exactly on, and one or a few units
in the last place around, bucket boundaries.  Every comparison is exact."""
import pytest
import torch

from oracle import tq_oracle as orc
from winnow_b200.cache import TurboQuantMSE, _get_quantizer
from winnow_b200.packed_backend import append_tokens
from winnow_b200.packing import unpack

pytestmark = pytest.mark.gpu
DEV = "cuda"


def check(x, bw):
    tq, oq = _get_quantizer(bw, 128, DEV, 42), orc.OracleQuantizer.get(bw, 128, 42)
    ref_idx, ref_norm = oq.quantize(x)
    idx, norm = tq.quantize(x.to(DEV))
    assert torch.equal(idx.cpu(), ref_idx) and torch.equal(norm.cpu(), ref_norm)
    packed, _ = tq.quantize(x.to(DEV), packed=True)
    assert torch.equal(unpack(packed, bw, 128).cpu(), ref_idx)


@pytest.mark.parametrize("rows", [6, 15, 16, 17, 63, 65, 2368, 2400, 5000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_vector_counts_and_types(rows, dtype):
    x = torch.randn(rows, 128, generator=torch.Generator().manual_seed(rows))
    x[:, ::61] *= 8.0
    check(x.to(dtype), 4)


@pytest.mark.parametrize("rows", [443, 444, 445, 447, 449, 464, 465, 592, 593])
def test_where_the_tensor_cores_take_over(rows):
    """Three vectors a multiprocessor (444 at 148), and the passes of 16 just above."""
    x = torch.randn(rows, 128, generator=torch.Generator().manual_seed(rows)).half()
    for bw in (3, 4, 8):
        check(x, bw)


@pytest.mark.parametrize("bw", [2, 3, 4, 5, 6, 8])
def test_widths_and_special_rows(bw):
    x = torch.randn(3000, 128, generator=torch.Generator().manual_seed(bw))
    x[1], x[2], x[3], x[4] = 0.0, x[2] * 1e-30, x[3] * 1e20, x[4] * 1e-12
    x[5] = 0.0
    x[5, 7] = -3.0                                     # one coordinate: codes follow a column of Pi
    check(x, bw)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("bw", [2, 4, 6, 8])
def test_zero_vectors_among_others(bw, dtype):
    """Vectors of zeros (of either sign) sit on the middle boundary exactly; vectors whose
    squares vanish, or with one element only, do not."""
    x = torch.randn(1200, 128, generator=torch.Generator().manual_seed(bw))
    x[::3] = 0.0
    x[3::9] = -0.0
    x[600:900] = 0.0                                    # whole passes
    x[601, 5], x[607, 127], x[613], x[640, 0] = 1e-23, -1e-30, 1e-25, 2.0
    check(x.to(dtype), bw)


def on_boundaries(bw):
    oq = orc.OracleQuantizer.get(bw, 128, 42)
    g = torch.Generator().manual_seed(99)
    edges = oq.boundaries
    y = torch.randn(4096, 128, generator=g, dtype=torch.float64) * 0.088
    pick = torch.randint(0, len(edges), (4096, 24), generator=g)
    inner = edges.double().abs() < 0.2
    pick = torch.where(inner[pick], pick, torch.full_like(pick, len(edges) // 2))
    y[:, :24] = edges.double()[pick] * (1 + torch.randint(-3, 4, (4096, 24), generator=g) * 2.0 ** -24)
    rest = (1.0 - (y[:, :24] ** 2).sum(1, keepdim=True)).clamp_min(1e-3).sqrt()
    y[:, 24:] *= rest / y[:, 24:].norm(dim=1, keepdim=True)          # |y| = 1: division leaves it in place
    return (y @ oq.Pi.double()).float()


@pytest.mark.parametrize("bw", [4, 8])
def test_coordinates_on_boundaries(bw):
    """x = y Pi with y on (or a few fp32 steps beside) boundaries: the rotation
    returns to within an ulp or so of them, on either side."""
    check(on_boundaries(bw), bw)


@pytest.mark.parametrize("longer", [0.0625, 3.0, 256.0, 4096.0])
@pytest.mark.parametrize("bw", [4, 8])
def test_matrix_with_rows_of_any_length(bw, longer):
    """Not a rotation: coordinates, boundaries and rounding errors all grow with the rows
    (4096: operands beyond fp16)."""
    x, oq, tq = on_boundaries(bw), orc.OracleQuantizer(bw, 128, 42), TurboQuantMSE(bw, 128, DEV)
    for t in (oq, tq):
        t.Pi, t.boundaries = (t.Pi * longer).contiguous(), (t.boundaries * longer).contiguous()
    idx, norm = tq.quantize(x.to(DEV))
    ref_idx, ref_norm = oq.quantize(x)
    assert torch.equal(idx.cpu(), ref_idx) and torch.equal(norm.cpu(), ref_norm)


def test_odd_strides_and_unaligned_destinations():
    g = torch.Generator().manual_seed(3)
    base = torch.randn(2, 4, 41, 131, generator=g)
    x = base[..., 1:129]                                # rows start at odd elements, stride 131
    check(x.to(torch.float32), 4)
    tq, oq = _get_quantizer(6, 128, DEV, 42), orc.OracleQuantizer.get(6, 128, 42)
    k, v = base.half()[..., 1:129], base.half()[..., 2:130]
    lens, S, P = [41, 50], 24, 8
    table = torch.tensor([[5, 0, 3], [1, 7, 2]], dtype=torch.int32)
    kp, vp = torch.zeros(P, 4, S, 96, dtype=torch.uint8), torch.zeros(P, 4, S, 96, dtype=torch.uint8)
    kn, vn = torch.zeros(P, 4, S, dtype=torch.float16), torch.zeros(P, 4, S, dtype=torch.float16)
    flat = torch.zeros(P * 4 * S * 96 + 3, dtype=torch.uint8, device=DEV)
    gk = flat[3:].view(P, 4, S, 96)                    # pages at an odd address
    gv, gkn, gvn = vp.to(DEV), kn.to(DEV), vn.to(DEV)
    append_tokens(k.to(DEV), v.to(DEV), gk, gkn, gv, gvn, table.to(DEV),
                  torch.tensor(lens, dtype=torch.int32, device=DEV), tq, tq)
    orc.append_tokens(kp, kn, vp, vn, table, [n - 41 for n in lens], k, v, oq, oq)
    assert torch.equal(gk.cpu(), kp) and torch.equal(gv.cpu(), vp)
    assert torch.equal(gkn.cpu(), kn) and torch.equal(gvn.cpu(), vn)
