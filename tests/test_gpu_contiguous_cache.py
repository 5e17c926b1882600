"""The contiguous cache beside its usual use: shapes that broadcast into its rings and
shapes that do not fit."""
import pytest
import torch

from oracle import tq_oracle as orc
from winnow_b200 import _lib
from winnow_b200.cache import TQPackedLayer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(B=4, H=2, D=128, n=9):
    g = torch.Generator().manual_seed(B)
    layer = TQPackedLayer(D, 4, DEV, 32)
    k, v = (torch.randn(B, H, n, D, generator=g).half().to(DEV) for _ in range(2))
    layer.update(k, v)
    return layer, k, v


@pytest.mark.parametrize("shape", [(1, 2, 3, 128), (4, 1, 3, 128), (1, 1, 3, 128)])
def test_one_sequence_or_head_goes_to_all(shape):
    layer, _, _ = _layer()
    x = torch.randn(shape, generator=torch.Generator().manual_seed(1)).half()
    k, v = layer.update(x.to(DEV), -x.to(DEV))
    o = orc.OracleQuantizer.get(4, 128, 42)
    for got, part in ((k, x), (v, -x)):
        idx, norm = o.quantize(part)
        ref = orc.dequantize_rows(orc.pack(idx, 4), norm.half(), o.centroids, o.Pi, 4, 128)
        assert got.shape == (4, 2, 12, 128)
        # fp16 outputs, one unit in the last place of the largest
        assert (got[:, :, 9:].float().cpu() - ref).abs().max() <= 2.0 ** -10 * ref.abs().max()


@pytest.mark.parametrize("shape", [(2, 2, 3, 128), (8, 2, 3, 128), (4, 3, 3, 128)])
def test_shapes_that_do_not_fit_raise(shape):
    layer, k, v = _layer()
    before = [t[:, :, :9].clone() for t in layer._k[:2] + layer._v[:2]]          # (the rest is uninitialised)
    x = torch.zeros(shape, dtype=torch.float16, device=DEV)
    with pytest.raises(RuntimeError):
        layer.update(x, x)
    assert layer.get_seq_length() == 9
    assert all(torch.equal(a, b[:, :, :9]) for a, b in zip(before, layer._k[:2] + layer._v[:2]))


def test_quantizer_on_another_device_raises():
    x = torch.zeros(2, 2, 3, 128, dtype=torch.float16, device=DEV)
    with pytest.raises(_lib.BackendError):
        TQPackedLayer(128, 4, "cpu", 32).update(x, x)
