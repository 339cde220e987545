"""The 16-bit heads-as-M kernel (64 heads and more) against the numpy oracle, where it can go wrong: the smallest and the
unequal head groups, quadrants without live rows, lengths around its 64-token tile and its 32-token share per CTA, every
kind of page, many short requests per CTA pair, and the sign of the softmax scale.
Tolerances as in test_decode_gpu.py: max-abs <= 2e-2, rel-L2 < 4e-3, natural-log LSE <= 1e-3."""
import math

import numpy as np
import pytest
import torch

import mla_oracle as O
import nvfp4_mla_b200 as mla
from nvfp4_mla_b200 import _lib, serving
from nvfp4_mla_b200.testing import SM_SCALE, SyntheticCache
from util import oracle_reference

pytestmark = pytest.mark.gpu
LN2 = math.log(2.0)


def run(c, sm_scale=SM_SCALE, num_splits=0, longest=1 << 20):
    # a high bound of the lengths selects the kernel, however short they are
    args = (c.q_nope, c.q_pe, c.ckv_cache, c.ckv_sf_cache, c.kpe_cache, c.page_table, c.kv_lens, sm_scale, c.ckv_scale, c.kpe_scale)
    out = mla.decode(*args, max_kv_len=longest, num_splits=num_splits)
    _, lse2 = mla.decode_partial(*args, max_kv_len=longest, num_splits=num_splits)
    assert mla.workspace_status() == 0
    return out.float().cpu().numpy(), lse2.cpu().numpy() * LN2


def check(c, sm_scale=SM_SCALE, num_splits=0, longest=1 << 20):
    got, lse = run(c, sm_scale, num_splits, longest)
    want, want_lse = oracle_reference(c, sm_scale)
    live = [b for b, n in enumerate(c.kv_lens_list) if n > 0]
    assert np.abs(got - want).max() <= 2e-2
    assert O.rel_l2(got[live], want[live]) < 4e-3
    assert np.abs(lse[live] - want_lse[live]).max() <= 1e-3
    for b, n in enumerate(c.kv_lens_list):
        if n == 0:
            assert (got[b] == 0).all() and np.isneginf(lse[b]).all()


@pytest.mark.parametrize("heads", [64, 80, 112, 128, 144, 192, 256])
@pytest.mark.parametrize("num_splits", [0, 3])
def test_head_groups(heads, num_splits):
    # (three hundred requests of up to 1500 tokens select the kernel; nearly all of them are three tokens long)
    check(SyntheticCache([1500, 513, 64, 1] + [3] * 296, 64, heads, None, None, seed=heads).to("cuda"), num_splits=num_splits, longest=1500)


@pytest.mark.parametrize("page_size", [1, 2, 8, 16, 32, 64, 256])
def test_lengths_around_the_tile(page_size):
    lens = [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 0, 191, 192, 193, 257]
    check(SyntheticCache(lens, page_size, 64, 0.5, 2.0, seed=page_size).to("cuda"))


def test_many_short_requests_per_pair():
    rng = np.random.default_rng(3)
    check(SyntheticCache([int(x) for x in rng.integers(1, 200, 300)], 16, 80, None, None, seed=5).to("cuda"))


@pytest.mark.parametrize("sm_scale", [-SM_SCALE, 0.0])
def test_sign_of_the_softmax_scale(sm_scale):
    check(SyntheticCache([300, 65], 64, 128, 0.5, 2.0, seed=9).to("cuda"), sm_scale)


def test_wide_range_of_query_magnitudes_and_non_finite_elements():
    c = SyntheticCache([500, 129], 64, 64, 0.01, 0.01, seed=2).to("cuda")
    c.q_nope[:, :, 7] *= 64.0                       # outlier channel
    c.q_nope[:, 3] *= 2.0 ** -60                    # a tiny row
    c.q_nope[:, 9] *= 2.0 ** -60
    c.q_pe[:, 9] *= 2.0 ** -60
    c.q_pe[:, 5] *= 32.0                            # the rope part decides the row's scale
    check(c)
    clean, _ = run(c)
    c.q_nope[0, 1, 11], c.q_nope[0, 2, 300], c.q_pe[1, 4, 3] = float("nan"), float("inf"), -float("inf")
    got, _ = run(c)
    assert np.isfinite(got).all()  # a non-finite element counts as 0
    hit = [(0, 1), (0, 2), (1, 4)]
    for b in range(2):
        for h in range(64):
            if (b, h) not in hit:
                assert np.array_equal(got[b, h], clean[b, h])
    c.q_nope[0, 1, 11], c.q_nope[0, 2, 300], c.q_pe[1, 4, 3] = 0.0, 0.0, 0.0
    zeroed, _ = run(c)
    assert np.array_equal(got, zeroed)


@pytest.mark.parametrize("q_len,heads", [(2, 32), (4, 16), (5, 16), (3, 64), (2, 128)])
@pytest.mark.parametrize("num_splits", [0, 2])
def test_several_query_tokens_in_one_pass(q_len, heads, num_splits):
    """Requests shorter than q_len, lengths around the tile (a tile that only the last tokens see), rows in two groups."""
    lens = [1500, 1, 2, 64, 65, 66, 129, 4, 640] + [7] * 191
    c = SyntheticCache(lens, 64, heads, 0.5, 2.0, seed=q_len).to("cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    q_nope = torch.randn(len(lens), q_len, heads, 512, generator=g, device="cuda").bfloat16()
    q_pe = torch.randn(len(lens), q_len, heads, 64, generator=g, device="cuda").bfloat16()
    assert _lib.load().nvfp4_mla_decode_multi_folds(len(lens), q_len, heads, max(lens), 0) == 1
    out = serving.decode_multi_token(q_nope, q_pe, c.ckv_cache, c.ckv_sf_cache, c.kpe_cache, c.page_table, c.kv_lens, SM_SCALE,
                                     c.ckv_scale, c.kpe_scale, max_kv_len=max(lens), num_splits=num_splits)
    assert mla.workspace_status() == 0
    for i in range(q_len):
        c.q_nope, c.q_pe = q_nope[:, i].contiguous(), q_pe[:, i].contiguous()
        c.kv_lens_list = [max(n - (q_len - 1 - i), 0) for n in lens]
        c.kv_lens = torch.tensor(c.kv_lens_list, dtype=torch.int32)
        want, _ = oracle_reference(c)
        got = out[:, i].float().cpu().numpy()
        live = [b for b, n in enumerate(c.kv_lens_list) if n > 0]
        assert np.abs(got - want).max() <= 2e-2 and O.rel_l2(got[live], want[live]) < 4e-3
        for b, n in enumerate(c.kv_lens_list):
            assert n > 0 or (got[b] == 0).all()


def test_both_sides_of_the_dispatch_agree():
    """The bound of the lengths chooses the kernel: 512 tokens the 16-head one, 2^20 this one."""
    c = SyntheticCache([400] * 10, 64, 64, None, None, seed=8).to("cuda")
    few, few_lse = run(c, longest=512)
    many, many_lse = run(c, longest=1 << 20)
    assert not np.array_equal(few, many)  # (they round differently: it is two kernels)
    assert O.rel_l2(few, many) < 4e-3 and np.abs(few_lse - many_lse).max() <= 1e-3


@pytest.mark.parametrize("page_size", [16, 64])
def test_page_ids_are_range_checked(page_size):
    c = SyntheticCache([200, 90], page_size, 128, None, None, seed=4).to("cuda")
    good, _ = run(c)
    c.page_table[1, 0] = c.ckv_cache.shape[0] + 5
    args = (c.q_nope, c.q_pe, c.ckv_cache, c.ckv_sf_cache, c.kpe_cache, c.page_table, c.kv_lens, SM_SCALE, c.ckv_scale, c.kpe_scale)
    out = mla.decode(*args, max_kv_len=1 << 20)
    assert mla.workspace_status(clear=True) == 3
    assert np.array_equal(out[0].float().cpu().numpy(), good[0]) and torch.isfinite(out.float()).all()


@pytest.mark.parametrize("power", [-30, -9, 12, 40])
def test_query_loaded_a_second_time_replaces_the_first(power):
    """Rows whose magnitude FP16 cannot hold as they are go through the query load twice, into the same places. A power of two in
    all queries, taken out again by the softmax scale, changes no bit of the result: the query's elements and their products with the
    ratio of the two scales (a power of two) are exact in either form."""
    c = SyntheticCache([1, 130, 7, 64] * 80, 64, 128, 0.5, 2.0, seed=6).to("cuda")
    c.q_nope, c.q_pe = (c.q_nope * 16).round() / 16, (c.q_pe * 16).round() / 16
    want, want_lse = run(c)
    c.q_nope *= 2.0 ** power
    c.q_pe *= 2.0 ** power
    for _ in range(5):
        got, lse = run(c, SM_SCALE * 2.0 ** -power)
        assert np.array_equal(got, want) and np.array_equal(lse, want_lse)


@pytest.mark.parametrize("top", [2.0 ** -8, 2.0 ** -2, 2.0 ** 6])
def test_small_query_elements_against_large_latents(top):
    """Half of the channels hold query elements 2^11 below the row's maximum, but meet latent values 2^17 above the others': they
    decide the scores (standard deviation about 3). Bound: rel-L2 < 4e-3 as elsewhere (the BF16 result alone is 1.7e-3); an error
    of 2^-25 of the row's maximum per element moves a score by less than 2^-13."""
    c = SyntheticCache([100, 64, 33] * 100, 64, 64, 4.0 / top, 1.0, seed=12).to("cuda")
    c.ckv_cache.random_(0, 256, generator=torch.Generator(device="cuda").manual_seed(2))  # all codes alike
    sf = c.ckv_sf_cache.view(torch.uint8)
    sf[..., :16], sf[..., 16:] = 0x7E, 0x01  # 448 and 2^-9
    c.q_nope[..., :256] *= top * 2.0 ** -11
    c.q_nope[..., 256:] = top
    c.q_pe.zero_()
    got, lse = run(c)
    want, want_lse = oracle_reference(c)
    assert O.rel_l2(got, want) < 4e-3 and np.abs(lse - want_lse).max() <= 1e-3


@pytest.mark.parametrize("block", [0, 9, 17, 31])  # (both parts of the tile, in either CTA)
def test_nan_scale_of_a_later_token_stays_out_of_earlier_query_tokens(block):
    """A foreign cache may hold a NaN block scale. In one pass for all query tokens a row that must not see the token multiplies its
    value with probability 0; the rows that do see it lose the partial result it is part of, as in a call of their own."""
    lens, q_len, heads = [7, 65, 130, 64] * 60, 4, 16
    c = SyntheticCache(lens, 64, heads, 0.5, 2.0, seed=3).to("cuda")
    g = torch.Generator(device="cuda").manual_seed(1)
    q_nope = torch.randn(len(lens), q_len, heads, 512, generator=g, device="cuda").bfloat16()
    q_pe = torch.randn(len(lens), q_len, heads, 64, generator=g, device="cuda").bfloat16()
    args = (q_nope, q_pe, c.ckv_cache, c.ckv_sf_cache, c.kpe_cache, c.page_table, c.kv_lens, SM_SCALE, c.ckv_scale, c.kpe_scale)
    assert _lib.load().nvfp4_mla_decode_multi_folds(len(lens), q_len, heads, 8192, 0) == 1
    clean = serving.decode_multi_token(*args, max_kv_len=8192)
    sf = c.ckv_sf_cache.view(torch.uint8)
    for b, n in enumerate(lens):  # the last token of half of the requests, the last but two of the others
        at = n - 1 if b % 8 < 4 else n - 3
        sf[c.page_table[b, at // 64], at % 64, block] = 0x7F if b % 2 else 0xFF
    out = serving.decode_multi_token(*args, max_kv_len=8192)
    for b in range(len(lens)):
        unaware = 3 if b % 8 < 4 else 1
        assert torch.equal(out[b, :unaware], clean[b, :unaware]), b
        if lens[b] <= 64:  # one partial result, lost
            assert not out[b, unaware:].any()


@pytest.mark.parametrize("heads,q_len", [(64, 1), (128, 1), (16, 4), (144, 1)])
def test_repeated_runs_give_the_same_bits(heads, q_len):
    """A race between the kernel's roles, or an issue warp that loses its operands, shows as results that come and go: many ragged requests
    (lengths from one token to fifty tiles), other batches in between, and every run equals the first bit for bit."""
    rng = np.random.default_rng(heads)
    lens = [int(x) for x in np.exp(rng.uniform(0, np.log(3200), 200))]
    c = SyntheticCache(lens, 16, heads, 0.5, 2.0, seed=heads, device="cuda")
    shape = (len(lens), q_len, heads)
    g = torch.Generator(device="cuda").manual_seed(1)
    q_nope, q_pe = torch.randn(*shape, 512, generator=g, device="cuda").bfloat16(), torch.randn(*shape, 64, generator=g, device="cuda").bfloat16()
    call = serving.decode_multi_token
    if q_len == 1:
        call, q_nope, q_pe = mla.decode, q_nope[:, 0], q_pe[:, 0]

    def once(n):
        return call(q_nope[:n], q_pe[:n], c.ckv_cache, c.ckv_sf_cache, c.kpe_cache, c.page_table[:n], c.kv_lens[:n], SM_SCALE, c.ckv_scale,
                    c.kpe_scale, max_kv_len=max(lens))

    first = {n: once(n) for n in (200, 173)}
    for i in range(60):
        for n, want in first.items():
            assert torch.equal(once(n), want), (i, n)
    assert mla.workspace_status() == 0
