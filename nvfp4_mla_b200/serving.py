"""The callers either side of the decode path, as a serving engine would use them: a paged latent-KV pool that appends
through the CUDA cache writer and decodes through the decode kernel, multi-token (speculative / MTP verify) decode, and
the W_UV projection after the latent output.

The reference lists these as what comes next around its kernel (README.md:88, 118-119, 414-415 of the reference
project): it has none of them, so there is no reference code to mirror; the arithmetic is the decode path's own and is
checked against the oracle per query position.
"""
import operator

import numpy as np
import torch

from . import _PRECISIONS, CKV, KPE, _append, _check_append, _decode, _lib, decode


def decode_multi_token(q_nope, q_pe, ckv_cache, ckv_sf_cache, kpe_cache, page_table, kv_lens, sm_scale,
                       ckv_scale=1.0, kpe_scale=1.0, max_kv_len=None, num_splits=0, precision="bf16"):
    """Decode ``Q`` query tokens per request against one cache (speculative or multi-token-prediction verify).

    ``q_nope [batch, Q, heads, 512]``, ``q_pe [batch, Q, heads, 64]``; ``kv_lens [batch]`` counts the tokens in the
    cache INCLUDING the ``Q`` new ones, which are its last ``Q`` positions. Query ``i`` attends causally to the first
    ``kv_lens - (Q - 1 - i)`` tokens. Returns ``[batch, Q, heads, 512]`` bfloat16.

    With ``precision="bf16"``, enough rows (``Q * heads`` of 64 and more) and enough tokens, all rows of a request share one
    pass over its cache: one call of the heads-as-M kernel, which cuts each row at its own length. Otherwise each query
    position runs as a request of its own that shares the original's pages (its row of the page table is repeated); the
    ``Q`` reads of a request's cache are scheduled next to each other and the later ones are served from L2. Either way the
    launch shape is fixed by ``max_kv_len``, and nothing synchronises if it is given (one read of the lengths if not).
    """
    if q_nope.dim() != 4 or q_pe.dim() != 4:
        raise RuntimeError("q_nope must be [batch, Q, heads, 512] and q_pe [batch, Q, heads, 64]")
    B, Q, H = q_nope.shape[:3]
    if tuple(q_pe.shape) != (B, Q, H, KPE) or q_nope.shape[3] != CKV:
        raise RuntimeError("q_nope must be [batch, Q, heads, 512] and q_pe [batch, Q, heads, 64]")
    if kv_lens.dim() != 1 or kv_lens.shape[0] != B or kv_lens.dtype != torch.int32:
        raise RuntimeError("kv_lens must be int32 [batch]")
    if Q > 1 and H > 0 and H % 16 == 0 and ckv_cache.is_cuda and _PRECISIONS.get(precision) == 0:
        if max_kv_len is None:
            max_kv_len = int(kv_lens.max()) if B else 0  # device sync; the lengths below are not longer
        with torch.cuda.device(ckv_cache.device):
            folds = _lib.load().nvfp4_mla_decode_multi_folds(B, Q, H, int(max_kv_len), 0)
        if folds == 1:
            out = _decode(q_nope.reshape(B, Q * H, CKV).contiguous(), q_pe.reshape(B, Q * H, KPE).contiguous(), ckv_cache, ckv_sf_cache,
                          kpe_cache, page_table.contiguous(), kv_lens.contiguous(), sm_scale, ckv_scale, kpe_scale, max_kv_len,
                          num_splits, 0, True, False, q_len=Q)[0]
            return out.view(B, Q, H, CKV)
    back = torch.arange(Q - 1, -1, -1, dtype=torch.int32, device=kv_lens.device)  # Q-1 .. 0 tokens not yet visible
    lens = (kv_lens[:, None] - back[None, :]).clamp_(min=0).reshape(B * Q).contiguous()
    table = page_table.repeat_interleave(Q, dim=0).contiguous()
    out = decode(q_nope.reshape(B * Q, H, CKV).contiguous(), q_pe.reshape(B * Q, H, KPE).contiguous(), ckv_cache,
                 ckv_sf_cache, kpe_cache, table, lens, sm_scale, ckv_scale, kpe_scale, max_kv_len, num_splits, precision)
    return out.view(B, Q, H, CKV)


class PagedLatentCache:
    """A fixed pool of NVFP4 latent-KV pages with per-request page lists: what a serving engine keeps per layer.

    Pages are handed out on the host (a free list), the page table and lengths live on the device, and every append
    goes through the CUDA cache writer. What a call has to tell the device (page ids, lengths, token positions) is put
    together on the host, which knows all of it, and crosses in one copy from pinned memory: no call waits for the GPU's work (the first copies of a
    size allocate pinned memory, which may). ``max_pages_per_request`` fixes the page-table width, ``max_kv_len`` the decode launch shape, so a decode step can be captured in a CUDA graph once the pages of the step have been reserved.
    """

    def __init__(self, num_pages, page_size, max_requests, max_pages_per_request, ckv_scale, kpe_scale, device="cuda"):
        dev = torch.device(device)
        self.page_size, self.ckv_scale, self.kpe_scale = page_size, float(ckv_scale), float(kpe_scale)
        self.ckv_cache = torch.zeros(num_pages, page_size, CKV // 2, dtype=torch.uint8, device=dev)
        self.ckv_sf_cache = torch.zeros(num_pages, page_size, CKV // 16, dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn)
        self.kpe_cache = torch.zeros(num_pages, page_size, KPE, dtype=torch.uint8, device=dev).view(torch.float8_e4m3fn)
        # page table and lengths share one array, so that an append updates both at once
        self._tables = torch.zeros(max_requests * (max_pages_per_request + 1), dtype=torch.int32, device=dev)
        self.page_table = self._tables[:max_requests * max_pages_per_request].view(max_requests, max_pages_per_request)
        self.kv_lens = self._tables[max_requests * max_pages_per_request:]
        self.max_kv_len = max_pages_per_request * page_size
        self._free = list(range(num_pages - 1, -1, -1))
        self._pages = [[] for _ in range(max_requests)]   # host mirror of the page lists
        self._lens = [0] * max_requests                   # host mirror of the lengths
        # the page table as the writer's page list: request r owns entries [r * width, (r + 1) * width)
        self._kv_indptr = torch.arange(0, (max_requests + 1) * max_pages_per_request, max(max_pages_per_request, 1),
                                       dtype=torch.int32, device=dev)

    @property
    def free_pages(self):
        return len(self._free)

    def release(self, request):
        """Returns the request's pages to the pool."""
        self._free.extend(reversed(self._pages[request]))
        self._pages[request], self._lens[request] = [], 0
        self.kv_lens[request].zero_()

    def append(self, requests, ckv, kpe):
        """Appends ``counts[i]`` new tokens to ``requests[i]``: ``requests`` is a list of ``(request, count)`` pairs and
        ``ckv [sum(counts), 512]`` / ``kpe [sum(counts), 64]`` (bfloat16) hold their latent rows in that order. A request may be
        named more than once: its shares follow each other. Whatever refuses the call does so before the pool changes."""
        if not requests:
            raise IndexError("append needs at least one request")
        width, known, free, n_free, page_size = self.page_table.shape[1], len(self._lens), self._free, len(self._free), self.page_size
        slots, values = [], []  # entries of the page table and of the lengths, and what they become
        reqs, counts, ends = [], [], []  # per entry of the call: request, tokens, the request's length after it
        grown, taken = {}, 0  # per request: [length, pages, new pages]; pages taken from the end of the free list
        for r, n in requests:
            if type(r) is not int or type(n) is not int or r < 0 or r >= known or n < 0:
                r, n = range(known)[r], operator.index(n)  # (a negative id counts from the end)
                if n < 0:
                    raise ValueError("counts must not be negative")
            to = grown.get(r)
            if to is None:
                to = grown[r] = [self._lens[r], len(self._pages[r]), []]
            end, held, fresh = to
            to[0] = end = end + n
            need = -(-end // page_size) - held
            if need > 0:
                if taken + need > n_free or held + need > width:
                    raise RuntimeError("out of cache pages")
                at = r * width + held
                slots += range(at, at + need)
                got = free[-taken - 1:-taken - need - 1:-1]
                values += got
                fresh += got
                to[1] = held + need
                taken += need
            reqs.append(r)
            counts.append(n)
            ends.append(end)
        slots += [known * width + r for r in grown]
        values += [to[0] for to in grown.values()]
        nnz, n_slots, counts, ends = sum(counts), len(slots), np.array(counts), np.array(ends)
        # position of token j of entry i: ends[i] - counts[i] + j
        first = np.cumsum(counts) - counts

        def fill(host):
            host[:8 * n_slots].view(np.int64)[:] = slots
            words = host[8 * n_slots:].view(np.int32)
            words[:n_slots] = values
            words[n_slots:n_slots + nnz] = np.repeat(reqs, counts)
            words[n_slots + nnz:] = np.arange(nnz) + np.repeat(ends - counts - first, counts)

        told = self._to_device(12 * n_slots + 8 * nnz, fill)
        words = told[8 * n_slots:].view(torch.int32)
        write = (ckv, kpe, words[n_slots:n_slots + nnz], words[n_slots + nnz:], self.ckv_cache, self.ckv_sf_cache, self.kpe_cache,
                 self.page_table.view(-1), self._kv_indptr)
        if _check_append(*write) and (ckv.data_ptr() % 16 or kpe.data_ptr() % 4):  # (the C entry would refuse that too late)
            raise RuntimeError("ckv must be 16-byte and kpe 4-byte aligned")
        self._tables.index_copy_(0, told[:8 * n_slots].view(torch.int64), words[:n_slots])
        _append(nnz, *write, self.ckv_scale, self.kpe_scale)
        del free[n_free - taken:]
        for r, (end, _, fresh) in grown.items():
            self._lens[r] = end
            self._pages[r] += fresh

    def _to_device(self, nbytes, fill):
        """A uint8 device copy of ``nbytes`` that ``fill`` writes into a host array, through one copy from pinned memory (the
        block returns to torch's host allocator, which hands it out again only after the copy has run)."""
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("a graph cannot capture this call: it would replay today's host data")
        staged = torch.empty(nbytes, dtype=torch.uint8, pin_memory=True)
        fill(staged.numpy())
        return staged.to(self.ckv_cache.device, non_blocking=True)

    def decode(self, requests, q_nope, q_pe, sm_scale, w_uv=None, precision="bf16"):
        """One decode step for ``requests`` (a list of request ids): ``q_nope [len(requests), heads, 512]``,
        ``q_pe [len(requests), heads, 64]``. Returns the latent output ``[n, heads, 512]``, or, with
        ``w_uv [heads, 512, v_head_dim]``, the value-space output ``[n, heads, v_head_dim]`` (the absorbed W_UV applied
        after attention)."""
        if precision not in _PRECISIONS:
            raise ValueError(f"precision must be one of {list(_PRECISIONS)}, got {precision!r}")
        longest = 0  # (the bound is the pool's capacity: by itself it would choose the kernel for long requests)
        if torch.is_tensor(requests):
            table, lens = self.page_table[requests.to(self.page_table.device)], self.kv_lens[requests.to(self.page_table.device)]
        else:
            if type(requests) is list and requests and all(type(r) is int for r in requests):  # (the usual form, without a tensor)
                ids = requests
            else:
                ids = torch.tensor(requests)
                if ids.dim() == 1 and ids.numel() and ids.dtype in (torch.int64, torch.int32):
                    ids = ids.tolist()
            if type(ids) is list:
                known = len(self._lens)
                if not (-known <= min(ids) and max(ids) < known):
                    raise IndexError("request id out of range")
                longest = max(1, max(self._lens[r] for r in ids))
                ids = np.array([r % known for r in ids], dtype=np.int64)
                idx = self._to_device(ids.nbytes, lambda host: host.__setitem__(slice(None), ids.view(np.uint8))).view(torch.int64)
                table, lens = self.page_table.index_select(0, idx), self.kv_lens.index_select(0, idx)
            else:  # a mask over all requests; what is neither ids nor a mask is refused by the indexing
                idx = ids.to(self.page_table.device)
                table, lens = self.page_table[idx].contiguous(), self.kv_lens[idx].contiguous()
        out = _decode(q_nope, q_pe, self.ckv_cache, self.ckv_sf_cache, self.kpe_cache, table, lens, sm_scale, self.ckv_scale, self.kpe_scale,
                      self.max_kv_len, 0, _PRECISIONS[precision], True, False, expected_kv_len=longest)[0]
        return out if w_uv is None else torch.einsum("bhc,hcv->bhv", out, w_uv.to(out.dtype))
