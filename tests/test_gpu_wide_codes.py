"""Quantizers and dequantizers on tensor cores at d = 96 and for codes of 5 and 6 bits: the packed bytes are those of the
reference-order kernels, norms and reconstructions at least as close to 64-bit arithmetic -- tile remainders, both sides of
the row count from which they are used, zero, tiny and huge rows, rows of a cache."""
import numpy as np
import pytest

import project_tensor_b200 as tg

pytestmark = pytest.mark.gpu

CASES = [("mse", 96, 1), ("mse", 96, 4), ("mse", 96, 6), ("mse", 64, 5), ("mse", 64, 6), ("mse", 128, 5), ("mse", 128, 6),
         ("prod", 96, 3), ("prod", 96, 4), ("prod", 96, 5), ("prod", 96, 6), ("prod", 64, 6), ("prod", 128, 6), ("prod", 96, 2)]


def _quantizer(kind, d, bits):
    return (tg.TurboQuantProd if kind == "prod" else tg.TurboQuantMSE)(d, bits, seed=2026, grid_size=4097, max_iter=64)


def _reconstruction64(quant, kind, enc):
    import torch
    mse = quant.mse if kind == "prod" else quant
    dev = enc.norms.device
    as64 = lambda a: torch.as_tensor(np.asarray(a), device=dev).double()
    out = as64(mse.codebook)[torch.as_tensor(enc.indices).long()] @ as64(mse.rotation)
    if kind == "prod":
        alpha = float(np.float32(np.sqrt(np.pi / 2) / quant.dimension))
        out = out + alpha * torch.as_tensor(enc.residual_norms).double()[:, None] * (torch.as_tensor(enc.qjl).double() @ as64(quant.projection))
    return out * torch.as_tensor(enc.norms).double()[:, None]


@pytest.mark.parametrize("kind,d,bits", CASES)
def test_packed_bytes_and_precision(lib_built, kind, d, bits):
    import torch
    quant = _quantizer(kind, d, bits)
    for n in (5328, 5329, 7104, 7105, 9473, 11841, 20001):
        x = torch.randn(n, d, device="cuda", generator=torch.Generator("cuda").manual_seed(n + d)) * 2.0
        x[3] = 0
        x[n - 1] *= 1e-20          # sum of squares below the tensor-core kernels' range
        x[n // 2] *= 1e4
        packed, restored, error = {}, {}, {}
        for path in ("auto", "exact"):
            quant.set_kernel_path(path)
            enc = quant.quantize(x)
            packed[path], restored[path] = tg.packed_buffers(enc), quant.dequantize(enc)
            want = _reconstruction64(quant, kind, enc)
            scale = want.norm(dim=1, keepdim=True).clamp_min(1e-300)          # (every row counts alike)
            error[path] = float(((restored[path].double() - want) / scale).norm() / (want / scale).norm())
        for name, exact in packed["exact"].items():
            if exact is None:
                continue
            if exact.dtype.is_floating_point:
                # norms: sums of d squares in another order (2 units in the last place); residual norms: the residual is down to 1/30 of the
                # unit vector, whose coordinates carry 1.5e-7
                bound = 5e-7 if name == "norms" else 5e-6
                assert float(((packed["auto"][name] - exact).abs() / exact.abs().clamp_min(1e-30)).max()) <= bound, (n, name)
            else:
                assert torch.equal(packed["auto"][name], exact), (n, name)
        # two roundings of the same float32 result differ by some 1.5e-7; no larger an error than the reference order's
        assert error["auto"] <= 1.1 * error["exact"] and error["auto"] <= 2.5e-7, (n, error)


@pytest.mark.parametrize("d,kbits,vbits", [(96, 4, 6), (128, 6, 5), (64, 6, 6)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
def test_rows_of_a_cache(lib_built, d, kbits, vbits, dtype):
    import torch
    kq, vq = _quantizer("prod", d, kbits), _quantizer("mse", d, vbits)
    groups, tokens = 3, 4001
    cache = tg.PackedKVCache(kq, vq, groups, tokens + 5)
    gen = torch.Generator("cuda").manual_seed(d)
    keys, values = (torch.randn(groups, tokens, d, device="cuda", generator=gen).to(getattr(torch, dtype)) for _ in range(2))
    cache.append(keys, values)
    want = tg.packed_buffers(kq.quantize(keys.float().reshape(-1, d)))
    have = cache.keys
    for name, rows in (("codes", have.codes), ("signs", have.signs)):
        rows = rows.view(groups, tokens + 5, -1)
        assert torch.equal(rows[:, :tokens].reshape(groups * tokens, -1), want[name].reshape(groups * tokens, -1)), name
        assert not bool(rows[:, tokens:].any()), name
    want = tg.packed_buffers(vq.quantize(values.float().reshape(-1, d)))
    assert torch.equal(cache.value_codes.view(groups, tokens + 5, -1)[:, :tokens].reshape(groups * tokens, -1),
                       want["codes"].reshape(groups * tokens, -1))


@pytest.mark.parametrize("kind,d,bits", [("mse", 96, 4), ("prod", 128, 6), ("mse", 64, 6)])
def test_without_scratch_the_reference_order_kernels_serve(lib_built, kind, d, bits):
    """A C caller that passes no scratch block for such a plan, which needed none before there was a kernel with lists."""
    import torch
    from project_tensor_b200 import _native
    lib, n = _native.load(), 12001
    quant = _quantizer(kind, d, bits)
    x = torch.randn(n, d, device="cuda", generator=torch.Generator("cuda").manual_seed(d))
    want = tg.packed_buffers(quant.quantize(x))
    plan, stream = quant._plans.handle(x.device), torch.cuda.current_stream().cuda_stream
    got = {k: torch.zeros_like(v) for k, v in want.items() if v is not None}
    if kind == "mse":
        _native.check(lib.tq_mse_quantize(plan, x.data_ptr(), n, got["codes"].data_ptr(), got["norms"].data_ptr(), None, 0, stream))
    else:
        _native.check(lib.tq_prod_quantize(plan, x.data_ptr(), n, got["codes"].data_ptr(), got["signs"].data_ptr(),
                                           got["residual_norms"].data_ptr(), got["norms"].data_ptr(), None, 0, stream))
    assert torch.equal(got["codes"], want["codes"])
    if kind == "prod":
        assert torch.equal(got["signs"], want["signs"])
