"""Errors of the fp16-split kernels against 64-bit results, from the unpacked codes: no larger than those of float32 multiply-adds.

The limits are what kernels that added float32 products in registers (one query: through tables of products), or hi and lo
products in accumulators of their own, gave for these inputs (2-norm of the error over 2-norm of the scores).  An accumulator that takes
every product at its full size, or bits whose mean is added back afterwards, exceeds them by 1.2 to 15 times."""
import math

import pytest

import project_tensor_b200 as tg

pytestmark = pytest.mark.gpu


def _randn(shape, seed):
    import torch
    return torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


def _keys64(quant, enc):
    import torch
    to64 = lambda a: torch.as_tensor(a, device="cuda").double()
    rows = to64(quant.mse.codebook)[enc.indices.long()] @ to64(quant.mse.rotation)
    rows += math.sqrt(math.pi / 2) / quant.dimension * enc.residual_norms.double()[:, None] * (enc.qjl.double() @ to64(quant.projection))
    return rows * enc.norms.double()[:, None]


_FEW = {64: 1.75e-7, 128: 2.6e-7, 256: 3.6e-7, 96: 2.75e-7}
_MANY = {64: 2.95e-7, 128: 4.4e-7, 256: 6.3e-7, 96: 2.75e-7}


@pytest.mark.parametrize("d", [64, 96, 128, 256])
@pytest.mark.parametrize("bits", [2, 3, 4, 5])
def test_scores(d, bits):
    n = 20011
    quant = tg.TurboQuantProd(d, bits, seed=2026)
    enc = quant.quantize(_randn((n, d), d + bits))
    keys = _keys64(quant, enc)
    few = {64: 2, 128: 4 if bits <= 4 else 2, 256: 1, 96: 1}[d]       # queries that the warp-level kernel takes
    for nq in (1, 2, 3, 4, 5, 16, 40):
        q = _randn((nq, d), nq)
        want = q.double() @ keys.T
        err = float((quant.attention_scores(q, enc).double() - want).norm() / want.norm())
        assert err <= (_FEW if nq <= few else _MANY)[d], (nq, err)
