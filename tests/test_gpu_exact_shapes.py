"""The reference-order kernels at the edges of their block shapes: one row, a row or two beyond a whole number of blocks,
the row counts around which another shape takes over, dimensions that are no multiple of the panels -- against
the oracle.  And the one-launch cache step for every element type."""
import numpy as np
import pytest

from oracle import turboquant_oracle as orc
import parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bits,counts", [
    (33, 3, (1, 149, 600)), (64, 5, (3, 592, 593, 4741)), (96, 6, (1, 148, 4739)), (100, 4, (5, 4740)),
    (128, 6, (2, 593, 4737)), (130, 2, (17, 1190)), (256, 5, (9, 1185, 4738)), (520, 3, (1, 33)),
])
def test_exact_kernels_reproduce_the_oracle_at_every_block_shape(lib_built, d, bits, counts):
    import project_tensor_b200 as tg
    prod = tg.TurboQuantProd(d, bits, seed=2026, grid_size=4097, max_iter=64)
    pp = orc.ProdParams(d, bits, orc.mse_params(d, prod.mse.bits, rotation=prod.mse.rotation, codebook=prod.mse.codebook),
                        prod.projection)
    prod.set_kernel_path("exact")
    for n in counts:
        x = (np.random.default_rng(d + n).standard_normal((n, d)) * 2.0).astype(np.float32)
        if n > 2:
            x[n // 2] = 0.0
        codes, qjl, rn, norms = orc.prod_quantize(pp, x)[:4]
        enc = prod.quantize(x)
        # one row and odd sizes take other BLAS kernels on the host, whose sums are ordered differently: a coordinate on a
        # knife edge may then differ, the floats in their last bits
        f, o, t = parity.code_flip_report(enc.indices, codes, prod.mse.rotation, prod.mse.boundaries, x)
        parity.assert_discrete_parity(f, o, t, f"codes, {n} rows")
        assert int((np.asarray(enc.qjl) != qjl).sum()) <= 1, n
        assert np.array_equal(enc.norms, norms), n
        assert parity.max_rel_scalar(enc.residual_norms, rn) <= 2e-6, n
        assert parity.max_rel_rows(prod.dequantize(enc), orc.prod_dequantize(pp, codes, qjl, rn, norms, (n,))) <= 5e-6, n


@pytest.mark.parametrize("d,groups,tokens", [(128, 64, 1), (64, 3, 5), (256, 7, 2), (96, 200, 3)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
def test_cache_step_in_one_launch_for_every_element_type(lib_built, d, groups, tokens, dtype):
    """Keys and values land behind the present rows, equal to quantize of the widened values; a full cache takes no more
    rows and its length stays at the capacity."""
    import torch
    import project_tensor_b200 as tg
    from project_tensor_b200 import _native
    kq, vq = tg.TurboQuantProd(d, 3, seed=2026), tg.TurboQuantMSE(d, 4, seed=77)
    kq.set_kernel_path("exact"), vq.set_kernel_path("exact")
    cap = 2 * tokens + 1
    cache = tg.PackedKVCache(kq, vq, groups, cap)
    gen = torch.Generator("cuda").manual_seed(d)
    keys = torch.randn((groups, cap + tokens, d), device="cuda", generator=gen).to(getattr(torch, dtype))
    values = torch.randn((groups, cap + tokens, d), device="cuda", generator=gen).to(getattr(torch, dtype))
    for step in range(2):
        part = slice(step * tokens, (step + 1) * tokens)
        cache.append(keys[:, part], values[:, part])
    assert cache.sync_length() == 2 * tokens
    # one step more than fits, past the Python check: the device drops what does not fit and saturates
    k, v = keys[:, 2 * tokens:3 * tokens].contiguous(), values[:, 2 * tokens:3 * tokens].contiguous()
    code = {"float32": _native.TQ_F32, "bfloat16": _native.TQ_BF16, "float16": _native.TQ_F16}[dtype]
    st = torch.cuda.current_stream().cuda_stream
    _native.check(_native.load().tq_kv_append(
        kq._plans.handle(cache.device), vq._plans.handle(cache.device), k.data_ptr(), v.data_ptr(), code, groups, tokens,
        cache.keys.codes.data_ptr(), cache.keys.signs.data_ptr(), cache.keys.residual_norms.data_ptr(),
        cache.keys.norms.data_ptr(), cache.value_codes.data_ptr(), cache.value_norms.data_ptr(), cap,
        cache.keys.length_device.data_ptr(), 1, st))
    assert int(cache.keys.length_device.item()) == min(3 * tokens, cap)
    filled = min(3 * tokens, cap)
    want_k = tg.packed_buffers(kq.quantize(keys[:, :filled].float()))
    want_v = tg.packed_buffers(vq.quantize(values[:, :filled].float()))
    for name, have in (("codes", cache.keys.codes), ("signs", cache.keys.signs), ("norms", cache.keys.norms),
                       ("residual_norms", cache.keys.residual_norms)):
        assert torch.equal(have.view(groups, cap, -1)[:, :filled], want_k[name].view(groups, filled, -1)), name
    assert torch.equal(cache.value_codes.view(groups, cap, -1)[:, :filled], want_v["codes"].view(groups, filled, -1))
    assert torch.equal(cache.value_norms.view(groups, cap)[:, :filled], want_v["norms"].view(groups, filled))


@pytest.mark.parametrize("d,bits,counts", [
    (64, 6, (4737, 9473)), (96, 6, (4737, 9473)), (128, 6, (4737, 7105, 8289)), (200, 4, (1185, 2369, 3553, 4737)),
    (300, 3, (592, 593, 1185, 2369)), (512, 4, (593, 1185, 2369)), (700, 3, (593, 1185)), (1024, 2, (593, 1185, 2369)),
])
def test_a_row_is_the_same_in_every_block_shape(lib_built, d, bits, counts):
    """One chain of multiply-adds per output in every shape: the bytes of a row do not depend on the rows beside it."""
    import torch
    import project_tensor_b200 as tg
    prod, mse = (make(d, bits, seed=2026, grid_size=4097, max_iter=64) for make in (tg.TurboQuantProd, tg.TurboQuantMSE))
    x = torch.randn((max(counts), d), device="cuda", generator=torch.Generator("cuda").manual_seed(d))
    for quant in (prod, mse):
        quant.set_kernel_path("exact")
        few = x[:3].contiguous(), x[-2:].contiguous()
        want = [(tg.packed_buffers(e), quant.dequantize(e)) for e in map(quant.quantize, few)]
        for n in counts:
            batch = torch.cat([x[:3], x[:n - 5], x[-2:]])
            enc = quant.quantize(batch)
            restored, packed = quant.dequantize(enc), tg.packed_buffers(enc)
            for part, (buffers, rows) in zip((slice(0, 3), slice(n - 2, n)), want):
                assert torch.equal(restored[part], rows), (n, part)
                for name, value in buffers.items():
                    assert value is None or torch.equal(packed[name][part], value), (n, part, name)


@pytest.mark.parametrize("d", [33, 64, 100, 128])
def test_two_rows_a_block_equal_one(lib_built, d):
    """More rows than SMs, up to two an SM, share blocks in pairs: the same bytes as in calls of at most 100 rows, an odd last row, zero
    rows on either side of a pair and the keys and values of a cache step included."""
    import torch
    import project_tensor_b200 as tg
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    prod, mse = (make(d, 4, seed=2026, grid_size=4097, max_iter=64) for make in (tg.TurboQuantProd, tg.TurboQuantMSE))
    x = torch.randn((2 * sms + 1, d), device="cuda", generator=torch.Generator("cuda").manual_seed(d)).bfloat16()
    x[4] = x[9] = 0
    ones = {}
    for quant in (prod, mse):
        parts = [tg.packed_buffers(quant.quantize(p.float())) for p in x.split(min(100, sms))]
        ones[quant] = {k: torch.cat([p[k] for p in parts]) for k, v in parts[0].items() if v is not None}
        for n in (sms + 1, 2 * sms - 1, 2 * sms, 2 * sms + 1):
            packed = tg.packed_buffers(quant.quantize(x[:n].float()))
            for name, want in ones[quant].items():
                assert torch.equal(packed[name], want[:n]), (n, name)
    for groups in (sms // 2 + 1, sms - 1, sms):
        cache = tg.PackedKVCache(prod, mse, groups, 1)
        cache.append(x[:groups], x[groups:2 * groups])
        for name in ("codes", "signs", "norms", "residual_norms"):
            assert torch.equal(getattr(cache.keys, name), ones[prod][name][:groups]), (groups, name)
        assert torch.equal(cache.value_codes, ones[mse]["codes"][groups:2 * groups])
        assert torch.equal(cache.value_norms, ones[mse]["norms"][groups:2 * groups]) and cache.sync_length() == 1
