"""Scores of one to four queries per group (and of one against so many keys that tables of its products are faster): tiles of 16 keys with a remainder, fewer tiles than warps, every code width, groups --
against q . dequantize(key) in 64-bit."""
import pytest

import project_tensor_b200 as tg
import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("bits", [2, 3, 4, 5])
def test_few_queries(d, bits):
    import torch
    quant = tg.TurboQuantProd(d, bits, seed=2026)
    gen = torch.Generator("cuda").manual_seed(d + bits)
    # where the table kernel takes over: many keys, many groups of few keys
    many = ((300, 1, 33), (151, 2, 256), (160, 1, 511), (150, 1, 256))
    many += ((1, 1, ((1 << 19) if bits <= 3 else (1 << 20)) + 33),) if d < 256 or bits <= 3 else ()
    for groups, qpg, n in many + ((1, 1, 1), (1, 1, 15), (3, 1, 4097), (1, 2, 17), (2, 2, 2368), (1, 3, 37889), (4, 4, 530), (1, 1, 300001)):
        keys = torch.randn(groups * n, d, device="cuda", generator=gen)
        keys[n // 2] = 0
        queries = torch.randn(groups * qpg, d, device="cuda", generator=gen) * 100
        queries[0] *= 1e-4
        enc = quant.quantize(keys)
        got = quant.attention_scores(queries, enc, groups=groups)
        want = torch.einsum("gqd,gnd->gqn", queries.view(groups, qpg, d).double(),
                            quant.dequantize(enc).double().view(groups, n, d)).reshape(groups * qpg, n)
        knorm = keys.norm(dim=1).view(groups, 1, n).expand(groups, qpg, n).reshape(groups * qpg, n)
        err = parity.max_score_err(got.cpu().numpy(), want.cpu().numpy(), queries.norm(dim=1)[:, None].cpu().numpy(),
                                   knorm.cpu().numpy(), d)
        assert err <= 2e-5, (groups, qpg, n, err)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("bits", [2, 4])
def test_queries_near_the_largest_float(d, bits):
    import torch
    quant = tg.TurboQuantProd(d, bits, seed=2026)
    gen = torch.Generator("cuda").manual_seed(d + bits)
    enc = quant.quantize(torch.randn(300, d, device="cuda", generator=gen) * 1e-3)
    queries = torch.randn(2, d, device="cuda", generator=gen)
    want = quant.attention_scores(queries, enc)
    for scale in (2.0 ** 116, 2.0 ** 121):       # (S q itself is near the largest float)
        got = quant.attention_scores(queries * scale, enc) * (1.0 / scale)
        assert float((got - want).abs().max()) <= 1e-6 * float(want.abs().max()), scale


@pytest.mark.parametrize("d,bits", [(64, 2), (64, 4), (128, 2), (128, 4), (256, 2), (256, 4)])
def test_one_query_on_both_sides_of_the_table_kernels_lines(d, bits):
    """Many groups with one or two blocks of keys each, and one group at the lowest count that takes tables."""
    import torch
    quant = tg.TurboQuantProd(d, bits, seed=2026)
    gen = torch.Generator("cuda").manual_seed(d + bits)
    for groups, qpg, n in ((888, 1, 33), (900, 1, 33), (900, 1, 128), (900, 1, 129), (900, 1, 256), (900, 1, 257), (900, 2, 250), (1, 1, (3 << 18) + 33)):
        if groups * n * d > 1 << 27:
            continue
        keys = torch.randn(groups * n, d, device="cuda", generator=gen)
        queries = torch.randn(groups * qpg, d, device="cuda", generator=gen) * 100
        enc = quant.quantize(keys)
        got = quant.attention_scores(queries, enc, groups=groups)
        want = torch.einsum("gqd,gnd->gqn", queries.view(groups, qpg, d).double(),
                            quant.dequantize(enc).double().view(groups, n, d)).reshape(groups * qpg, n)
        knorm = keys.norm(dim=1).view(groups, 1, n).expand(groups, qpg, n).reshape(groups * qpg, n)
        err = float(((got.double() - want).abs() / (queries.norm(dim=1)[:, None] * knorm)).max())
        # (the reconstruction and the score are each within a few 1e-6 of the product of the norms)
        assert err <= 1e-5, (groups, qpg, n, err)
