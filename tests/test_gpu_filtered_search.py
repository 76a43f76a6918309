"""Top-k search through the single-fp16 first stage (tq_score_filter.cu): the result is the stable sort of the full-accuracy
score matrix, at the smallest key counts it serves, with ragged ends, for one and several passes of queries, for data its
lists have no room for and for keys and queries its bound does not cover."""
import pytest

pytestmark = pytest.mark.gpu


def _fell_back(prod, enc, q, k):
    """Whether a search over up to 4,194,304 keys went on to the score matrix: it lies over the lists of the first stage in the scratch
    block and is larger than they are (32 queries and more), so that its end is written by nothing else."""
    import torch
    import project_tensor_b200 as tg
    from project_tensor_b200 import _native
    lib, packed, n = _native.load(), tg.packed_buffers(enc), enc.prefix_shape[0]
    handle, nq = prod._plans.handle(q.device), q.shape[0]
    need = lib.tq_topk_scratch_bytes(handle, 1, nq, n, k)
    scratch = torch.full((need,), 0xA5, dtype=torch.uint8, device=q.device)
    top_s, top_i = torch.empty((nq, k), device=q.device), torch.empty((nq, k), dtype=torch.int64, device=q.device)
    _native.check(lib.tq_score_batched(handle, q.data_ptr(), 1, nq, packed["codes"].data_ptr(), packed["signs"].data_ptr(),
                                       packed["residual_norms"].data_ptr(), packed["norms"].data_ptr(), n, None, k, top_s.data_ptr(),
                                       top_i.data_ptr(), 0, scratch.data_ptr(), need, torch.cuda.current_stream().cuda_stream))
    end = 4 * n * nq // 100 * 98
    return not bool((scratch[end - (1 << 20):end] == 0xA5).all())


def _check(prod, enc, q, k, rows=None):
    import torch
    prod.set_kernel_path("tensor")       # one to four queries would take a lookup-table kernel, with other last bits
    mat = prod.attention_scores(q, enc)
    prod.set_kernel_path("auto")
    top_s, top_i = prod.attention_scores(q, enc, topk=k, index_base=2)
    srt = torch.sort(mat, dim=1, descending=True, stable=True)
    for r in range(q.shape[0]) if rows is None else rows:
        assert torch.equal(top_s[r], srt.values[r, :k]) and torch.equal(top_i[r], srt.indices[r, :k] + 2), r


@pytest.mark.parametrize("d,bits,n,nq,k", [
    (128, 4, 1 << 20, 32, 100), (128, 4, (1 << 20) + 77, 64, 100), (128, 2, (1 << 21) + 1, 3, 1000), (64, 3, (1 << 20) + 129, 33, 10),
    (64, 5, (1 << 21) + 64, 17, 64), (256, 4, (1 << 20) + 5, 40, 50), (256, 2, (1 << 21) + 3, 5, 100), (128, 5, (1 << 20) + 1, 100, 20),
])
def test_filtered_search_equals_the_sorted_matrix(lib_built, d, bits, n, nq, k):
    import torch
    import project_tensor_b200 as tg
    gen = torch.Generator("cuda").manual_seed(n + d)
    x = torch.randn((n, d), device="cuda", generator=gen) * (0.1 + 3.0 * torch.rand((n, 1), device="cuda", generator=gen))
    x[n // 3] = 0.0
    q = torch.randn((nq, d), device="cuda", generator=gen) * torch.logspace(-3, 3, nq, device="cuda")[:, None]
    prod = tg.TurboQuantProd(d, bits, seed=2026)
    _check(prod, prod.quantize(x), q, k)


@pytest.mark.parametrize("d,n,nq,k", [(128, (1 << 20) + 11, 32, 100), (64, (1 << 20) + 64, 70, 10), (256, (1 << 20) + 3, 33, 20), (64, (1 << 22) + 77, 70, 20)])
def test_filtered_search_falls_back_when_its_lists_are_too_short(lib_built, d, n, nq, k):
    """Half the keys are one vector: more exact ties at the threshold than a round has room for.  One pass of queries and several, with
    the procedures of up to 4,194,304 keys and of more behind the first stage."""
    import torch
    import project_tensor_b200 as tg
    gen = torch.Generator("cuda").manual_seed(5)
    x = torch.randn((n, d), device="cuda", generator=gen)
    x[1000:1000 + n // 2] = x[7]
    q = torch.randn((nq, d), device="cuda", generator=gen)
    q[3] = x[7]
    q[4] = 0.0           # every score is zero
    prod = tg.TurboQuantProd(d, 4, seed=2026)
    enc = prod.quantize(x)
    _check(prod, enc, q, k)
    if nq == 32:
        assert _fell_back(prod, enc, q, k)


@pytest.mark.parametrize("n", [(1 << 20) + 5, 1 << 21])
def test_filtered_search_for_queries_without_a_score(lib_built, n):
    """NaN queries: every score is NaN, and the first rows are the best.  The other queries are unharmed."""
    import torch
    import project_tensor_b200 as tg
    gen = torch.Generator("cuda").manual_seed(7)
    prod = tg.TurboQuantProd(64, 4, seed=2026)
    enc = prod.quantize(torch.randn((n, 64), device="cuda", generator=gen))
    q = torch.randn((33, 64), device="cuda", generator=gen)
    q[5, 3] = float("nan")
    _check(prod, enc, q, 10, rows=[0, 4, 6, 32])
    top_s, top_i = prod.attention_scores(q, enc, topk=10)
    assert bool(top_s[5].isnan().all()) and top_i[5].tolist() == list(range(10))


@pytest.mark.parametrize("n", [(1 << 20) + 5, 1 << 22])
def test_keys_without_a_score_rank_as_in_a_selection_from_the_matrix(lib_built, n):
    """NaN norms: such scores come first up to 4,194,304 keys, the lowest rows first.  More of them than a query wants, and fewer."""
    import torch
    import project_tensor_b200 as tg
    gen = torch.Generator("cuda").manual_seed(8)
    prod = tg.TurboQuantProd(64, 4, seed=2026)
    enc = prod.quantize(torch.randn((n, 64), device="cuda", generator=gen))
    tg.packed_buffers(enc)["norms"][3::n // 16] = float("nan")
    q = torch.randn((32, 64), device="cuda", generator=gen)
    prod.set_kernel_path("tensor")
    srt = torch.sort(prod.attention_scores(q, enc), dim=1, descending=True, stable=True)      # (NaN sorts as the greatest)
    prod.set_kernel_path("auto")
    for k in (10, 40):
        top_s, top_i = prod.attention_scores(q, enc, topk=k)
        assert torch.equal(top_i, srt.indices[:, :k])
        assert torch.equal(top_s.nan_to_num(nan=7e30), srt.values[:, :k].nan_to_num(nan=7e30))


def test_scores_that_are_nearly_all_minus_infinity(lib_built):
    """Finite norms and products below the smallest float: some thirty scores of each query are finite, fewer than one in the sample."""
    import torch
    import project_tensor_b200 as tg
    n, k = (1 << 20) + 5, 100
    gen = torch.Generator("cuda").manual_seed(9)
    prod = tg.TurboQuantProd(64, 4, seed=2026)
    enc = prod.quantize(torch.randn((n, 64), device="cuda", generator=gen))
    q = torch.randn((1, 64), device="cuda", generator=gen).expand(32, 64) * 1e6
    packed = tg.packed_buffers(enc)
    packed["residual_norms"][:] = 0.0
    packed["norms"][:] = torch.where(prod.attention_score(q[0], enc) < 0, 1e37, -1e37)
    prod.set_kernel_path("tensor")
    mat = prod.attention_scores(q, enc)
    prod.set_kernel_path("auto")
    assert 5 <= int(torch.isfinite(mat[0]).sum()) < k
    srt = torch.sort(mat, dim=1, descending=True, stable=True)
    top_s, top_i = prod.attention_scores(q, enc, topk=k)
    assert torch.equal(top_s, srt.values[:, :k]) and torch.equal(top_i, srt.indices[:, :k])


def test_scratch_of_a_search_is_that_of_one_score_matrix(lib_built):
    import torch
    import project_tensor_b200 as tg
    from project_tensor_b200 import _native
    handle = tg.TurboQuantProd(128, 4, seed=2026)._plans.handle(torch.device("cuda", 0))
    for queries in (1, 16, 64, 1000, 10000):
        for keys in (1 << 20, 1 << 21, 1 << 22):
            got = _native.load().tq_topk_scratch_bytes(handle, 1, queries, keys, 20)
            # a float per query and key; lists of every 65,536 keys, prepared queries and (few queries) gathered keys behind it
            assert got <= queries * keys * 4 + queries * (keys >> 16) * 20 * 8 + (32 << 20), (queries, keys)


def test_filtered_search_lists_keys_its_bound_does_not_cover(lib_built):
    """Hand-made norms: huge residual norms (the scaled sign operand leaves the fp16 range), huge and negative norms; few enough
    for the lists, which a whole warp's keys enter beside a key of huge norm."""
    import torch
    import project_tensor_b200 as tg
    d, n, nq, k = 128, (1 << 20) + 3, 32, 100
    gen = torch.Generator("cuda").manual_seed(6)
    prod = tg.TurboQuantProd(d, 4, seed=2026)
    enc = prod.quantize(torch.randn((n, d), device="cuda", generator=gen))
    packed = tg.packed_buffers(enc)
    packed["residual_norms"][5::n // 40] = 1.0e7
    packed["norms"][11::n // 50] *= -50.0
    packed["norms"][1013::n // 20] = 1.0e12
    q = torch.randn((nq, d), device="cuda", generator=gen)
    _check(prod, enc, q, k)
    top_s, top_i = prod.attention_scores(q, enc, topk=k)
    for first, step in ((5, n // 40), (1013, n // 20)):       # they are among the best, and the first stage has seen to it
        assert all(bool(((row - first) % step == 0).any()) for row in top_i)
    assert not _fell_back(prod, enc, q, k)
