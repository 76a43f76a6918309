"""Errors of the fp16-split kernels against 64-bit results, from the unpacked codes: no larger than those of float32 multiply-adds.

The limits are what kernels that added float32 products in registers (one query: through tables of products), or hi and lo
products in accumulators of their own, gave for these inputs (2-norm of the error over 2-norm of the scores).  An accumulator that takes
every product at its full size, or bits whose mean is added back afterwards, exceeds them by 1.2 to 15 times."""
import math

import pytest

import project_tensor_b200 as tg
from project_tensor_b200.cache import PackedKVCache

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


def _values64(quant, enc):
    import torch
    to64 = lambda a: torch.as_tensor(a, device="cuda").double()
    return to64(quant.codebook)[enc.indices.long()] @ to64(quant.rotation) * enc.norms.double()[:, None]


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


@pytest.mark.parametrize("d,kbits,vbits,groups,n", [(64, 4, 3, 16, 129), (64, 4, 4, 4, 30011), (128, 4, 4, 4, 30011), (128, 2, 2, 16, 1531),
                                                    (128, 5, 1, 4, 30011)])
def test_attention(d, kbits, vbits, groups, n):
    """Exponents of about 10 rounded to float32 alone give some 5e-7; the weighted sums must not add a bias to it."""
    import torch
    kq, vq = tg.TurboQuantProd(d, kbits, seed=2026), tg.TurboQuantMSE(d, vbits, seed=77)
    cache = PackedKVCache(kq, vq, groups, (n + 15) // 16 * 16)
    loud = torch.ones(d, device="cuda")
    loud[3::d // 4] = 10.0
    cache.append(_randn((groups, n, d), 1) * loud, _randn((groups, n, d), 2) * loud)
    for qpg in (1, 4, 8):
        q = _randn((groups, qpg, d), qpg)
        got, square = cache.attend(q).double(), []
        for g in range(groups):
            s = (q[g].double() @ _keys64(kq, cache.keys.encoding(g)).T) * d ** -0.5
            want = torch.softmax(s, dim=-1) @ _values64(vq, cache.value_encoding(g))
            square.append(((got[g] - want).norm(dim=1) / want.norm(dim=1)).square())
        assert float(torch.cat(square).mean().sqrt()) <= 1.5e-6, qpg


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("scale", [300.0, 1e-4])
def test_codebooks_of_any_size(d, scale):
    """The parts of a centroid have a unit of their own, so that a plan's codebook may lie outside [-1, 1]."""
    import torch
    from project_tensor_b200.turboquant import _PlanSet
    n, kq, vq = 3001, tg.TurboQuantProd(d, 4, seed=2026), tg.TurboQuantMSE(d, 4, seed=77)
    cache = PackedKVCache(kq, vq, 1, 3008)
    cache.append(_randn((1, n, d), 1), _randn((1, n, d), 2))
    for quant in (kq.mse, vq):
        quant.codebook = quant.codebook * scale
    kq._plans = cache.keys._plans = _PlanSet(d, 3, kq.mse.rotation, kq.mse.codebook, kq.projection)
    vq._plans = cache._vplans = _PlanSet(d, 4, vq.rotation, vq.codebook, None)
    keys, q = _keys64(kq, cache.keys.encoding(0)), _randn((1, 2, d), 3)
    want = q[0].double() @ keys.T
    err = float((kq.attention_scores(q[0], cache.keys.encoding(0)).double() - want).norm() / want.norm())
    assert err <= _FEW[d], err
    for qpg in (2, 5):
        q = _randn((1, qpg, d), qpg)
        small = min(1.0, 1.0 / scale)
        w = torch.softmax((q[0].double() @ keys.T) * small * d ** -0.5, dim=-1) @ _values64(vq, cache.value_encoding(0))
        got = cache.attend(q, scale=small * d ** -0.5)[0].double()
        assert float((got - w).norm() / w.norm()) <= 1.5e-6, qpg
