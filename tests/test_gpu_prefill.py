"""Bulk appends to a key/value cache: rows of every element type go straight into place, and are what the quantizers give
for the widened rows -- tile remainders, a cache that is partly filled, bit widths without a tensor-core kernel."""
import pytest

import project_tensor_b200 as tg
from project_tensor_b200.cache import PackedKVCache

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16", "float16"])
@pytest.mark.parametrize("d,kbits,vbits,groups,lengths", [
    (128, 3, 4, 3, (5, 4001)),           # 12,003 rows: a tile with 99 of them
    (64, 4, 3, 4, (1500, 1190, 7)),      # the second call has 4,760 rows, just above what one launch takes
    (128, 6, 2, 2, (2500,)),             # 5-bit keys have no tensor-core kernel, the values do
    (96, 4, 4, 1, (4200,)), (256, 4, 4, 2, (3000,)),
    (256, 6, 4, 2, (3000, 7)),           # the same at d = 256; the second call reads the length the first one raised
])
def test_bulk_append_equals_quantize(dtype, d, kbits, vbits, groups, lengths):
    import torch
    kq = tg.TurboQuantProd(d, kbits, seed=2026, grid_size=4097, max_iter=64)
    vq = tg.TurboQuantMSE(d, vbits, seed=77, grid_size=4097, max_iter=64)
    cap = sum(lengths) + 3
    cache = PackedKVCache(kq, vq, groups, cap)
    gen = torch.Generator("cuda").manual_seed(d + kbits)
    keys, values = (torch.randn(groups, sum(lengths), d, device="cuda", generator=gen).to(getattr(torch, dtype)) for _ in range(2))
    keys[0, 1] = 0
    keys[0, 2] *= 1e-4
    at = 0
    for n in lengths:
        cache.append(keys[:, at:at + n].contiguous(), values[:, at:at + n].contiguous())
        at += n
        assert len(cache) == at and int(cache.keys.length_device.item()) == at
    want = tg.packed_buffers(kq.quantize(keys.float().reshape(-1, d)))
    kc = cache.keys
    for name, have in (("codes", kc.codes), ("signs", kc.signs), ("norms", kc.norms), ("residual_norms", kc.residual_norms)):
        have = have.view(groups, cap, -1)
        assert torch.equal(have[:, :at].reshape(groups * at, -1), want[name].reshape(groups * at, -1)) or (
            "norms" in name and float((have[:, :at].reshape(-1) / want[name].reshape(-1) - 1).nan_to_num().abs().max()) <= 1e-6), name
        assert not bool(have[:, at:].any()), name
    want = tg.packed_buffers(vq.quantize(values.float().reshape(-1, d)))
    assert torch.equal(cache.value_codes.view(groups, cap, -1)[:, :at].reshape(groups * at, -1), want["codes"].reshape(groups * at, -1))
    assert float((cache.value_norms.view(groups, cap)[:, :at].reshape(-1) / want["norms"] - 1).abs().max()) <= 1e-6


@pytest.mark.parametrize("d", [128, 256])
def test_bulk_append_of_values_alone_raises_the_length(d):
    import torch
    from project_tensor_b200 import _native
    lib = _native.load()
    vq = tg.TurboQuantMSE(d, 4, seed=77, grid_size=4097, max_iter=64)
    n, cap, dev = 6000, 6400, torch.device("cuda", 0)
    values = torch.randn(1, n, d, device=dev, generator=torch.Generator("cuda").manual_seed(d))
    plan, stream = vq._plans.handle(dev), torch.cuda.current_stream().cuda_stream
    codes = torch.zeros((cap, d // 2), dtype=torch.uint8, device=dev)
    norms, length = torch.zeros(cap, device=dev), torch.full((1,), 100, dtype=torch.int64, device=dev)
    need = lib.tq_kv_prefill_scratch_bytes(None, plan, n)
    scratch = torch.empty(need, dtype=torch.uint8, device=dev)
    _native.check(lib.tq_kv_prefill(None, plan, None, values.data_ptr(), _native.TQ_F32, 1, n, None, None, None, None,
                                    codes.data_ptr(), norms.data_ptr(), cap, 100, length.data_ptr(), scratch.data_ptr(), need, stream))
    assert int(length.item()) == 100 + n
    want = tg.packed_buffers(vq.quantize(values[0]))
    assert torch.equal(codes[100:100 + n], want["codes"]) and torch.equal(norms[100:100 + n], want["norms"])


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("d,tokens,offset", [(100, 1, 100), (20, 7, 20), (64, 1, 3), (128, 2500, 1), (256, 2500, 5)])
def test_append_takes_16_bit_rows_off_a_16_byte_boundary(dtype, d, tokens, offset):
    import torch
    kq, vq = tg.TurboQuantProd(d, 3, seed=2026, grid_size=4097, max_iter=64), tg.TurboQuantMSE(d, 4, seed=77, grid_size=4097, max_iter=64)
    groups = 2
    gen = torch.Generator("cuda").manual_seed(d)
    flat = torch.randn(groups * tokens * d + offset, device="cuda", generator=gen).to(getattr(torch, dtype))
    rows = flat[offset:].view(groups, tokens, d)
    assert rows.data_ptr() % 16 != 0 and rows.is_contiguous()
    for keys, values in ((rows, rows), (rows, rows.clone()), (rows.clone(), rows)):
        cache = PackedKVCache(kq, vq, groups, tokens + 1)
        cache.append(keys, values)
        want = PackedKVCache(kq, vq, groups, tokens + 1)
        want.append(rows.float(), rows.float())
        for have, other in ((cache.keys, want.keys), (cache, want)):
            for name in ("codes", "signs", "norms", "residual_norms", "length_device") if have is cache.keys else ("value_codes", "value_norms"):
                assert torch.equal(getattr(have, name), getattr(other, name)), name
