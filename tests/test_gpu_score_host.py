"""attention_score of one NumPy query, which goes through one call into the library: the scores of the device path, whatever the
query's type, layout and shape, from several threads and streams at a time, and nothing of a kernel that gave up."""
import threading

import numpy as np
import pytest

import project_tensor_b200 as tg
from project_tensor_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,bits", [(64, 4), (128, 3), (96, 6), (256, 4), (40, 2)])
def test_scores_are_those_of_the_device_path(d, bits):
    import torch
    quant = tg.TurboQuantProd(d, bits, seed=2026, grid_size=4097, max_iter=64)
    rng = np.random.default_rng(d)
    for n in (2, 255, 4096, 16384, 16385):
        enc = quant.quantize(rng.standard_normal((n, d)).astype(np.float32))
        q = rng.standard_normal(d)
        want = quant.attention_score(torch.from_numpy(q.astype(np.float32)).cuda(), enc).cpu().numpy()
        for form in (q.astype(np.float32), q, q.astype(np.float32)[None, :], np.repeat(q.astype(np.float32), 2)[::2]):
            got = quant.attention_score(form, enc)
            assert isinstance(got, np.ndarray) and got.dtype == np.float32 and got.shape == (n,) and np.array_equal(got, want), n
    enc = quant.quantize(rng.standard_normal((6, 7, d)).astype(np.float32))
    assert quant.attention_score(q, enc).shape == (6, 7)
    enc.prefix_shape = (7, -1)
    assert quant.attention_score(q, enc).shape == (7, 6)
    for bad in (np.zeros(d + 1, np.float32), np.zeros((2, d), np.float32), np.float32(1)):
        with pytest.raises(ValueError):
            quant.attention_score(bad, enc)


def test_threads_and_streams_have_blocks_of_their_own():
    import torch
    quant = tg.TurboQuantProd(64, 4, seed=2026)
    rng = np.random.default_rng(5)
    enc = quant.quantize(rng.standard_normal((3000, 64)).astype(np.float32))
    queries = rng.standard_normal((12, 40, 64)).astype(np.float32)
    want = [[quant.attention_score(q, enc) for q in mine] for mine in queries]
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for q, w in zip(queries[k], want[k]):
                if not np.array_equal(quant.attention_score(q, enc), w):
                    wrong.append(k)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_a_kernel_that_gave_up_is_reported():
    import torch
    quant = tg.TurboQuantProd(128, 4, seed=2026)
    rng = np.random.default_rng(6)
    x = torch.from_numpy(rng.standard_normal((6000, 128)).astype(np.float32)).cuda()
    q = rng.standard_normal(128).astype(np.float32)
    want = quant.attention_score(q, quant.quantize(x))
    quant._plans.set_wait_limit(0)           # the first wait that finds its barrier unfinished counts as run out
    enc = quant.quantize(x)
    quant._plans.set_wait_limit(4_000_000_000)
    with pytest.raises(_native.TurboQuantNativeError, match="gave up"):
        quant.attention_score(q, enc)
    assert np.array_equal(quant.attention_score(q, quant.quantize(x)), want)
