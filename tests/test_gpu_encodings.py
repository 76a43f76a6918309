"""Encodings whose ``prefix_shape`` was edited."""

import numpy as np
import pytest

import project_tensor_b200 as tg

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
