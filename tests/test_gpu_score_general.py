"""Score matrices at dimensions and bit widths without a tensor-core kernel: every code width, dimensions that end inside a sign
word, key and query counts around the block's, groups -- against q . dequantize(key) in 64-bit."""
import numpy as np
import pytest

import project_tensor_b200 as tg
import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bits", [(96, 6), (33, 3), (96, 2), (100, 4), (48, 5), (256, 6), (260, 7), (64, 8), (72, 9), (1024, 3), (2, 3)])
def test_matrix_of_any_geometry(d, bits):
    import torch
    quant = tg.TurboQuantProd(d, bits, seed=2026, grid_size=4097, max_iter=64)
    gen = torch.Generator("cuda").manual_seed(d + bits)
    for n, nq in ((1, 1), (129, 2), (511, 3), (513, 8), (1025, 9), (40001, 17)) if d < 1000 else ((700, 9),):
        keys = torch.randn(n, d, device="cuda", generator=gen)
        queries = torch.randn(nq, d, device="cuda", generator=gen)
        enc = quant.quantize(keys)
        got = quant.attention_scores(queries, enc)
        want = queries.double() @ quant.dequantize(enc).double().T
        err = parity.max_score_err(got.cpu().numpy(), want.cpu().numpy(), queries.norm(dim=1)[:, None].cpu().numpy(),
                                   keys.norm(dim=1)[None, :].cpu().numpy(), d)
        assert got.shape == (nq, n) and err <= 2e-5, (n, nq, err)
    one = quant.attention_score(queries[0], enc)
    assert np.allclose(one.cpu().numpy(), got[0].cpu().numpy(), rtol=0, atol=2e-5 * float(got.abs().max()))
