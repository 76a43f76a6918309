"""What a call leaves behind besides its result: encodings whose ``prefix_shape`` was edited, the counter of rows done in the reference's
order."""
import ctypes

import numpy as np
import pytest

import project_tensor_b200 as tg
from project_tensor_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["numpy", "cuda", "cpu"])
def test_edited_prefix_shape(lib_built, kind):
    import torch
    d, n = 64, 24
    x = np.random.default_rng(1).standard_normal((n, d)).astype(np.float32)
    as_kind = {"numpy": lambda a: a, "cuda": lambda a: torch.from_numpy(a).cuda(), "cpu": torch.from_numpy}[kind]
    mse, prod = tg.TurboQuantMSE(d, 3, seed=5), tg.TurboQuantProd(d, 3, seed=5)
    for quant in (mse, prod):
        enc = quant.quantize(as_kind(x))
        flat = quant.dequantize(enc)
        for prefix, shape in (((2, -1), (2, 12)), ((-1,), (24,)), ((4, 3, 2), (4, 3, 2))):
            enc.prefix_shape = prefix
            got = quant.dequantize(enc)
            assert tuple(got.shape) == shape + (d,) and bool((got.reshape(n, d) == flat).all())
            if quant is prod:
                assert tuple(quant.attention_score(as_kind(x[0]), enc).shape) == shape
        for prefix in ((5, 5), (-1, -1), (-4, -6), (7, -1)):
            enc.prefix_shape = prefix
            with pytest.raises((ValueError, RuntimeError)):
                quant.dequantize(enc)


def test_rows_done_in_reference_order_are_those_of_the_last_call(lib_built):
    import torch
    prod, rows, dev = tg.TurboQuantProd(128, 4, seed=5), ctypes.c_int64(-1), torch.device("cuda", 0)
    for n in (200_000, 300, 5):
        prod.quantize(torch.randn(n, 128, device=dev, generator=torch.Generator(dev).manual_seed(n)))
        _native.check(_native.load().tq_plan_last_recheck_rows(prod._plans.handle(dev), torch.cuda.current_stream().cuda_stream, ctypes.byref(rows)))
        assert rows.value == n if n < 1000 else 0 < rows.value < n // 50
