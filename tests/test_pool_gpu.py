"""The paged pool's bookkeeping on the device against its host mirror: page-crossing appends, ragged counts, zero counts, a
request named twice, release and reuse of pages, and what it refuses."""
import numpy as np
import pytest
import torch

import mla_oracle as O
import nvfp4_mla_b200 as mla
from nvfp4_mla_b200 import serving

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("page_size", [1, 16, 64])
def test_appends_land_where_the_page_table_says(page_size):
    rng = np.random.default_rng(page_size)
    pool = serving.PagedLatentCache(700, page_size, 5, 400, 0.5, 2.0)
    rows = {r: [] for r in range(5)}
    for step in [[(0, 3), (3, 0), (4, 130)], [(3, 1), (0, 64)], [(2, 65), (1, 1), (0, 1)], "release 0", [(0, 40), (4, 2)]]:
        if step == "release 0":
            pool.release(0)
            rows[0] = []
            continue
        n = sum(c for _, c in step)
        ckv = torch.from_numpy(rng.standard_normal((n, 512), dtype=np.float32)).bfloat16()
        kpe = torch.from_numpy(rng.standard_normal((n, 64), dtype=np.float32)).bfloat16()
        at = 0
        for r, c in step:
            rows[r] += list(ckv[at:at + c])
            at += c
        pool.append(step, ckv.cuda(), kpe.cuda())
        table, lens, cache = pool.page_table.cpu(), pool.kv_lens.cpu(), pool.ckv_cache.cpu()
        for r in range(5):
            assert int(lens[r]) == len(rows[r]) == pool._lens[r]
            assert table[r, :len(pool._pages[r])].tolist() == pool._pages[r]
            if rows[r]:
                t = torch.arange(len(rows[r]))
                packed, _ = O.quantize_ckv(torch.stack(rows[r]).float().numpy(), 0.5)
                assert np.array_equal(cache[table[r][t // page_size].long(), t % page_size].numpy(), packed)


def test_refusals():
    pool = serving.PagedLatentCache(4, 16, 2, 3, 0.5, 2.0)
    z = lambda n: (torch.zeros(n, 512, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, 64, dtype=torch.bfloat16, device="cuda"))
    with pytest.raises(IndexError):
        pool.append([], *z(0))
    with pytest.raises(RuntimeError, match="out of cache pages"):
        pool.append([(0, 49)], *z(49))
    with pytest.raises(RuntimeError, match="batch_indices"):
        pool.append([(1, 3)], *z(4))
    pool.append([(1, 3)], *z(3))
    q = torch.zeros(1, 16, 512, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 16, 64, dtype=torch.bfloat16, device="cuda")
    for bad in (2, -3):
        with pytest.raises(IndexError):
            pool.decode([bad], *q, 0.1)
    assert torch.equal(pool.decode([1], *q, 0.1), pool.decode(torch.tensor([-1]), *q, 0.1))


def test_a_request_named_twice_gets_its_shares_one_after_the_other():
    """The pool's bytes, tables and lengths equal those of a pool that appended the shares in calls of their own."""
    g = torch.Generator(device="cuda").manual_seed(7)
    steps = [[(0, 3), (0, 2)], [(1, 20), (0, 14), (1, 1), (0, 30)], [(-3, 1), (0, 0), (0, 2)]]
    pools = [serving.PagedLatentCache(20, 16, 3, 8, 0.5, 2.0) for _ in range(2)]
    for step in steps:
        n = sum(c for _, c in step)
        ckv, kpe = torch.randn(n, 512, generator=g, device="cuda").bfloat16(), torch.randn(n, 64, generator=g, device="cuda").bfloat16()
        pools[0].append(step, ckv, kpe)
        at = 0
        for r, c in step:
            pools[1].append([(r, c)], ckv[at:at + c], kpe[at:at + c])
            at += c
    assert state(pools[0]) == state(pools[1]) and pools[0]._lens == [52, 21, 0]
    for name in ("ckv_cache", "ckv_sf_cache", "kpe_cache"):
        a, b = (getattr(p, name).view(torch.uint8) for p in pools)
        assert torch.equal(a, b) and int(a.count_nonzero())


def state(pool):
    return (list(pool._free), [list(p) for p in pool._pages], list(pool._lens), pool.page_table.cpu().tolist(), pool.kv_lens.cpu().tolist())


@pytest.mark.parametrize("why", ["pages", "width", "id", "count", "rows", "dtype", "alignment", "capture"])
def test_a_refused_append_leaves_the_pool_unchanged(why):
    """Also where an earlier request of the same call could have been served: nothing of it may stay behind on the host, whose
    next append would tell the device only what it believes to be new."""
    pool = serving.PagedLatentCache(7, 16, 3, 4, 0.5, 2.0)
    rows = lambda n, dtype=torch.bfloat16: (torch.zeros(n, 512, dtype=dtype, device="cuda"), torch.zeros(n, 64, dtype=dtype, device="cuda"))
    pool.append([(2, 20)], *rows(20))
    before = state(pool)
    requests, given, error = [(0, 17), (1, 33)], rows(50), RuntimeError
    if why == "pages":
        requests, given = [(0, 33), (1, 33)], rows(66)
    elif why == "width":
        requests, given = [(0, 17), (2, 45)], rows(62)
    elif why == "id":
        requests, given, error = [(0, 17), (3, 1)], rows(18), IndexError
    elif why == "count":
        requests, given, error = [(0, 17), (1, -1)], rows(16), ValueError
    elif why == "rows":
        requests, given = [(0, 17), (1, 5)], rows(21)
    elif why == "dtype":
        requests, given = [(0, 17), (1, 5)], rows(22, torch.float32)
    elif why == "alignment":
        requests, given = [(0, 17), (1, 5)], (torch.zeros(22 * 512 + 4, dtype=torch.bfloat16, device="cuda")[4:].view(22, 512), rows(22)[1])
    else:
        requests, given = [(0, 17), (1, 5)], rows(22)
    torch.cuda.synchronize()
    if why == "capture":
        with pytest.raises(error), torch.cuda.graph(torch.cuda.CUDAGraph()):
            pool.append(requests, *given)
    else:
        with pytest.raises(error):
            pool.append(requests, *given)
    assert state(pool) == before
    pool.append([(0, 17), (1, 5)], *rows(22))  # what fits is served as if nothing had happened
    assert pool._lens == [17, 5, 20] == pool.kv_lens.tolist() and pool.free_pages == 2
    for r in range(3):
        assert pool.page_table[r, :len(pool._pages[r])].tolist() == pool._pages[r]
    assert len(sum(pool._pages, [])) == len(set(sum(pool._pages, []))) == 5


def test_forms_of_request_ids():
    """Whole numbers in any container, or a mask over all requests; anything else is refused and not read as a number."""
    pool = serving.PagedLatentCache(8, 16, 2, 3, 0.5, 2.0)
    g = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda").bfloat16()
    pool.append([(0, 5), (1, 20)], r(25, 512), r(25, 64))
    q = r(1, 16, 512), r(1, 16, 64)
    want = pool.decode([1], *q, 0.1)
    for ids in ((1,), np.array([1]), np.array([1], dtype=np.int32), [False, True], np.array([False, True]), [torch.tensor(1, device="cuda")],
                torch.tensor([1]), torch.tensor([1], device="cuda"), torch.tensor([False, True])):
        assert torch.equal(pool.decode(ids, *q, 0.1), want), ids
    for ids in ([1.7], [1.0], [], np.array([1.0])):
        with pytest.raises(IndexError):
            pool.decode(ids, *q, 0.1)


def test_decode_runs_the_kernel_of_the_lengths_and_not_of_the_capacity():
    """A pool of long requests that holds short ones: the bits are those of a call whose bound is the longest request (the 16-head
    kernel), not those of a call with the capacity as its bound. Lengths that a program advances on the device by itself are served
    in full all the same (rel-L2 < 4e-3 between two kernels of the 16-bit mode, as in the other tests)."""
    pool = serving.PagedLatentCache(40, 64, 8, 4096, 0.5, 2.0)
    g = torch.Generator(device="cuda").manual_seed(4)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda").bfloat16()
    lens = [40, 300, 5, 130, 77, 200, 1, 290]
    pool.append(list(enumerate(lens)), r(sum(lens), 512), r(sum(lens), 64))
    q = r(8, 64, 512), r(8, 64, 64)

    def decode(bound):
        return mla.decode(*q, pool.ckv_cache, pool.ckv_sf_cache, pool.kpe_cache, pool.page_table, pool.kv_lens, 0.07, 0.5, 2.0, max_kv_len=bound)

    got = pool.decode(list(range(8)), *q, 0.07)
    assert torch.equal(got, decode(300)) and not torch.equal(got, decode(pool.max_kv_len))
    pool.kv_lens += 300 * (pool.kv_lens == 300).int()  # (past the request's pages: page 0's rows, for both)
    pool.kv_lens += 1
    got, want = pool.decode(list(range(8)), *q, 0.07).float(), decode(pool.max_kv_len).float()
    assert O.rel_l2(got.cpu().numpy(), want.cpu().numpy()) < 4e-3
    with pytest.raises(ValueError, match="precision"):
        pool.decode([0], q[0][:1], q[1][:1], 0.07, precision="fp4")
