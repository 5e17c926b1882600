"""A dequantisation kernel whose waits run out says so instead of handing out rows it never
wrote.  The waits are told to give up at once; nothing is left running."""
import pytest
import torch

from winnow_b200 import _lib
from winnow_b200.cache import TQPackedCache, _get_quantizer, dequantize_rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def give_up():
    L = _lib.lib()
    yield lambda: L.wtq_dequant_wait_tries(0)
    L.wtq_dequant_wait_tries(-1)
    torch.cuda.synchronize()
    L.wtq_dequant_gave_up()


@pytest.mark.parametrize("rows", [1, 130, 148 * 128 * 5])
@pytest.mark.parametrize("mode,dtype", [(None, torch.bfloat16), ("tc", torch.float32), ("tc_fast", torch.float16)])
def test_next_call_or_question_reports_it(give_up, rows, mode, dtype):
    L, tq = _lib.lib(), _get_quantizer(4, 128, DEV, 42)
    g = torch.Generator().manual_seed(rows)
    codes = torch.randint(0, 256, (rows, 64), generator=g, dtype=torch.uint8).to(DEV)
    norms = (torch.rand(rows, generator=g) + 0.5).half().to(DEV)

    def call():
        out = torch.zeros(rows, 128, dtype=dtype, device=DEV)
        return dequantize_rows(codes, norms, tq.centroids, tq.Pi, 4, 128, out=out, mode=mode)

    good = call()
    torch.cuda.synchronize()
    assert L.wtq_dequant_gave_up() == 0
    give_up()
    bad = call()
    torch.cuda.synchronize()
    L.wtq_dequant_wait_tries(-1)
    assert not bad.any()                                  # no row was written
    with pytest.raises(_lib.BackendError, match="gave up"):
        call()
    assert torch.equal(call(), good) and L.wtq_dequant_gave_up() == 0      # once
    give_up()
    call()
    L.wtq_dequant_wait_tries(-1)
    torch.cuda.synchronize()
    assert L.wtq_dequant_gave_up() == 1 and torch.equal(call(), good)


def test_contiguous_cache_check(give_up):
    cache = TQPackedCache(128, 4, DEV, 64, 2)
    x = torch.randn(2, 2, 5, 128, generator=torch.Generator().manual_seed(1)).half().to(DEV)
    for layer in range(2):
        cache.update(x, x, layer)
    cache.check()
    give_up()
    cache.update(x, x, 1)
    with pytest.raises(_lib.BackendError):
        cache.check()
    _lib.lib().wtq_dequant_wait_tries(-1)
    cache.update(x, x, 0)
    cache.check()
