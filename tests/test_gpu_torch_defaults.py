"""Results do not depend on torch's default dtype and default device, which belong to the user's program."""
import numpy as np
import pytest

import project_tensor_b200 as tg

pytestmark = pytest.mark.gpu


def _everything(quant, x, q):
    import torch
    enc = quant.quantize(x)
    out = {k: v.cpu().numpy() for k, v in tg.packed_buffers(enc).items()}
    out["restored"], out["one"], out["many"] = quant.dequantize(enc), quant.attention_score(q[0], enc), quant.attention_scores(q, enc)
    out["pairs"] = quant.attention_score(x, enc)
    out["top_scores"], out["top_indices"] = quant.attention_scores(q, enc, topk=5)
    on_device = quant.quantize(torch.from_numpy(x).to("cuda"))
    out["device"] = quant.attention_scores(torch.from_numpy(q).to("cuda"), on_device).cpu().numpy()
    host = tg.quantize_to_host(quant, x)
    out.update({"host_" + k: v.numpy() for k, v in host.items()})
    return out


@pytest.mark.parametrize("name", ["float64", "bfloat16"])
def test_default_dtype_and_device(lib_built, name):
    import torch
    quant = tg.TurboQuantProd(64, 4, seed=2026)
    rng = np.random.default_rng(3)
    x, q = rng.standard_normal((250, 64)).astype(np.float32), rng.standard_normal((8, 64)).astype(np.float32)
    want = _everything(quant, x, q)
    try:
        torch.set_default_dtype(getattr(torch, name))
        torch.set_default_device("cuda")
        got = _everything(quant, x, q)
    finally:
        torch.set_default_device(None)
        torch.set_default_dtype(torch.float32)
    assert want.keys() == got.keys()
    for key in want:
        assert got[key].dtype == want[key].dtype and np.array_equal(got[key], want[key]), key
