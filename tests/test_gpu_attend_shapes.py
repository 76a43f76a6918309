"""Decode attention at the edges of its tiles (16 keys a warp, 12 warps a block, four or eight queries a pass), for every pair of
bit widths, and with value norms whose weights leave the fp16 range unless their scale follows them -- against the
composition of the package's scoring and dequantize kernels with a 64-bit softmax."""
import pytest

import project_tensor_b200 as tg
from project_tensor_b200.cache import PackedKVCache

pytestmark = pytest.mark.gpu


def _randn(shape, seed):
    import torch
    return torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


def _check(d, kbits, vbits, qpg, counts, grow=0.0):
    import torch
    groups = 2
    kq, vq = tg.TurboQuantProd(d, kbits, seed=2026), tg.TurboQuantMSE(d, vbits, seed=77)
    queries = _randn((groups, qpg, d), 5)
    for n in counts:
        cache = PackedKVCache(kq, vq, groups, (n + 15) // 16 * 16)
        values = _randn((groups, n, d), 7)
        if grow:      # norms from 10^-grow to 10^grow, up the one group and down the other
            power = torch.linspace(-grow, grow, n, device="cuda")
            values = values * torch.stack([10.0 ** power, 10.0 ** power.flip(0)])[:, :, None]
        cache.append(_randn((groups, n, d), 6), values)
        got = cache.attend(queries).double()
        for g in range(groups):
            s = kq.attention_scores(queries[g], cache.keys.encoding(g)).double() * d ** -0.5
            want = torch.softmax(s, dim=-1) @ vq.dequantize(cache.value_encoding(g)).double()
            assert float((got[g] - want).abs().max()) <= 3e-5 * float(want.abs().max()), (n, g)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kbits", [2, 3, 4, 5])
@pytest.mark.parametrize("vbits", [1, 2, 3, 4])
def test_every_pair_of_widths(d, kbits, vbits):
    _check(d, kbits, vbits, 4, (1, 193))
    _check(d, kbits, vbits, 9, (47,))


@pytest.mark.parametrize("qpg", [1, 5, 8])
def test_tile_and_block_edges(qpg):
    _check(128, 3, 4, qpg, (15, 16, 17, 191, 192, 385, 6157))


@pytest.mark.parametrize("grow", [6.0, 17.0])
def test_value_norms_far_apart(grow):
    _check(128, 4, 4, 4, (700, 5000), grow)
    _check(64, 3, 2, 6, (700,), grow)


@pytest.mark.parametrize("d", [64, 128])
def test_length_word_of_an_append_at_work(d):
    """While an append runs on another stream, the bits above the length count its blocks: they are not part of the length."""
    import torch
    groups, n, cap = 2, 300, 512
    cache = PackedKVCache(tg.TurboQuantProd(d, 4, seed=2026), tg.TurboQuantMSE(d, 4, seed=77), groups, cap)
    cache.append(_randn((groups, n, d), 6), _randn((groups, n, d), 7))
    queries = _randn((groups, 3, d), 5)
    want = cache.attend(queries)
    cache.keys.length_device += 37 << 40
    assert cache.sync_length() == n
    for got in (cache.attend(queries), cache.attend(queries, use_device_length=True)):
        assert float((got - want).abs().max()) <= 1e-5 * float(want.abs().max())
    cache.keys.length_device.fill_(-1)
    assert not bool(cache.attend(queries, use_device_length=True).any())
