// Weight-absorbed MLA decode for many query rows per request, 16-bit mode, with the query rows (heads) as the M dimension
// of both MMAs. The 16-head kernel (mla_decode_vt_sm100.cuh) converts a token once per 16 heads; here one FP16 copy of a
// token serves up to 128 rows:
//
//   HBM --L2 prefetch, 16-byte loads--> convert warps' registers --> K/V tile in smem, FP16, [token][channel], 128-byte swizzle
//   QK^T : S[row, token] = Q[row, 576] . K^T    A = Q (FP16) from tensor memory (latent 0..255, rope) / smem (latent 256..511),
//                                               B = the K/V tile read K-major, N = 64 tokens
//   PV   : O[row, chan] += P[row, token] . V    A = P (FP16) from tensor memory, written there by the softmax threads,
//                                               B = the same K/V tile read MN-major, N = 256 channels, K = 16 tokens
// Both K and V are exact in FP16 (e2m1 x e4m3 has six significant bits), Q is exact after a power-of-two scaling of the
// row (a BF16 has eight), the accumulators are fp32.
//
// O for 128 rows x 512 channels would need all 512 tensor-memory columns, so a PAIR of CTAs (a cluster of two) shares a
// request: both compute the full scores, CTA `cg` accumulates channels [256 cg, 256 cg + 256). CTA `cg` dequantises
// tokens [32 cg, 32 cg + 32) of every 64-token tile into its own tile and sends the same bytes to its peer's tile with
// bulk copies through distributed shared memory. The pair is one unit of the schedule and writes one partial slot.
//
// What bounds it from below is the tensor pipe. Per 64-token tile and CTA 20 MMAs of 32 cycles (A in tensor memory), 16 of
// 48 (A in shared memory, bound by the operand read) and 4 of 128 for PV: 1920 cycles. Storage allows two K/V tiles only
// (Q 144 KB, O 128 KB and S / P 48 KB of tensor memory + shared memory leave room for 2.2), so a tile is handed over in two
// parts: A = the nine panels minus this CTA's PV half (free as soon as QK^T has read them), B = the four panels PV reads.
// The next tile's part A is converted and multiplied while PV of the previous tile still holds part B.
//
// Measured, 128 heads, two requests of 1M tokens: 981 us a call against 1725 with the 16-head kernel (eight groups).
//
// Tensor memory (512 columns): Q latent 0..255: 0..127 | Q rope: 128..159 | S: 160..223 | P: 224..255 | O: 256..511.
// Warp roles (640 threads): 0-7 softmax + query load + epilogue, 8-15 dequantise (warp = 64-channel panel), 16 QK^T
// issue, 17 L2 prefetch (at the end it also waits for the peer's last buffer releases, so that no CTA leaves while its
// peer may still signal it), 18 PV issue. Every wait is bounded (ptx::mbar_wait).
#pragma once
#include "mla_decode_sm100.cuh"

namespace mla {

constexpr int kH16Threads = 640;
constexpr int kH16Rows = 128;              // query rows per CTA pair = MMA M (at most; the rest of M is dead)
constexpr int kH16Tile = 64;               // tokens per tile
constexpr int kH16Own = kH16Tile / 2;      // token rows one CTA of the pair loads and converts per tile
constexpr int kH16Panel = kH16Tile * 128;  // one 64-channel panel of the FP16 tile
constexpr int kH16Ahead = 6;               // tiles between a load and its L2 prefetch
constexpr uint32_t kH16PeerA = 4 * 4096 + 8 * 512, kH16PeerB = 4 * 4096;  // bytes the peer sends per tile, parts A and B

struct H16Smem {
  alignas(1024) uint8_t q[4][kH16Rows * 128];   // latent channels 256..511 of Q, FP16, row = query row, four panels of 64 channels
  alignas(1024) uint8_t kv[2][9][kH16Panel];    // panels 0..7: latent channels, panel 8: rope
  Seg segs[kSegBatch];
  alignas(8) uint64_t full_a[2], full_b[2];     // part of the tile in place: local convert warps + the peer's bytes
  // buffer part released, by CTA x of the pair (each CTA keeps the releases of both): part A by its QK^T, part B by its PV
  uint64_t free_a[2][2], free_b[2][2];          // [x][buffer]
  uint64_t s_full, s_free;                      // one phase per tile
  uint64_t p_full, pv_done;                     // one phase per tile
  uint64_t q_full;                              // query of the segment in place (8 softmax warps)
  float xch[2][kH16Rows], xl[2][kH16Rows];      // softmax pairs: maxima / sums exchanged between a quadrant's two warps
  volatile uint32_t progress;                   // tiles converted so far: paces the L2 prefetch
  uint32_t tmem_base;
  int abort_flag;
};
constexpr size_t h16_smem_bytes() { return sizeof(H16Smem) + 1024; }

struct H16Cols {
  static constexpr uint32_t QN = 0, QR = 128, S = 160, P = 224, O = 256;
};

// tiles of a segment: its 128-token units cut at the last live token
__device__ __forceinline__ int h16_tiles(const Seg& g) {
  if (g.ntiles <= 0) return 0;
  const int live = (g.tok_end - g.tok0 + kH16Tile - 1) / kH16Tile;
  return live < 2 * g.ntiles ? live : 2 * g.ntiles;
}

// ---------------------------------------------------------------------------------------------------------------
// role: L2 prefetch of this CTA's token rows (lane = row), kH16Ahead tiles ahead of the convert warps. Paced by a counter
// and not by a barrier's phases: nothing waits for this warp, so it may fall any number of tiles behind.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ bool h16_wait_converted(H16Smem& s, uint32_t tiles) {
  if (s.progress >= tiles) return true;
  const long long t0 = clock64();
  while (s.progress < tiles) {
    if (*static_cast<volatile int*>(&s.abort_flag) || clock64() - t0 > ptx::kWaitLimitCycles) return false;
    __nanosleep(100);
  }
  return true;
}
__device__ __forceinline__ void h16_prefetch_rows(const DecodeParams& P, const Seg& seg, int t, int cg, int lane) {
  const int tok = seg.tok0 + t * kH16Tile + kH16Own * cg + lane;
  if (tok >= seg.tok_end) return;
  const int page = P.page_table[(long long)seg.b * P.pt_stride + (tok >> P.page_shift)];
  if (uint32_t(page) >= uint32_t(P.num_pages)) return;
  const int in_page = tok & ((1 << P.page_shift) - 1);
  const long long row = ((long long)page << P.page_shift) + in_page;
  ptx::prefetch_l2(P.ckv + row * 256), ptx::prefetch_l2(P.ckv + row * 256 + 128);
  if ((lane & 1) == 0 || in_page == 0) ptx::prefetch_l2(P.kpe + row * 64);
  if ((lane & 3) == 0 || in_page == 0) ptx::prefetch_l2(P.sf + row * 32);
}
__device__ __forceinline__ void h16_prefetch_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, int cg) {
  const int lane = ptx::lane_id();
  for (int si = 0; si < n_segs; ++si) {
    const Seg seg = s.segs[si];
    const int nt = h16_tiles(seg);
    if (nt <= 0) continue;
    if (it == 0)
      for (int t = 1; t < kH16Ahead && t < nt; ++t) h16_prefetch_rows(P, seg, t, cg, lane);
    const int t_next = nt > kH16Ahead ? nt - kH16Ahead : 0;
    for (int t = 0; t < nt; ++t, ++it) {
      if (!__all_sync(~0u, h16_wait_converted(s, it))) return;
      if (t + kH16Ahead < nt) h16_prefetch_rows(P, seg, t + kH16Ahead, cg, lane);
      if (t == t_next)  // the next segment's query rows and first tiles
        for (int sj = si + 1; sj < n_segs; ++sj) {
          const Seg nx = s.segs[sj];
          const int nn = h16_tiles(nx);
          if (nn <= 0) continue;
          const int r0 = nx.hg * P.heads_per_cta, nr = P.heads - r0 < P.heads_per_cta ? P.heads - r0 : P.heads_per_cta;
          const long long row0 = (long long)nx.b * P.heads + r0;
          for (int i = lane; i < nr * 9; i += 32)
            ptx::prefetch_l2(i < nr * 8 ? reinterpret_cast<const char*>(P.q_nope + row0 * CKV) + i * 128
                                        : reinterpret_cast<const char*>(P.q_pe + row0 * KPE) + (i - nr * 8) * 128);
          for (int t2 = 0; t2 < kH16Ahead && t2 < nn; ++t2) h16_prefetch_rows(P, nx, t2, cg, lane);
          break;
        }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// role: dequantise (8 warps) this CTA's 32 token rows of every tile, into its own tile and the peer's. Warp w: panel w
// (64 channels); a lane takes half a panel row (16 packed bytes = two scale blocks) of rows lane / 2 and 16 + lane / 2,
// so that a warp's load touches 16 lines and its 16-byte stores are conflict-free. Rope: rows 4 w .. 4 w + 3, eight lanes
// per row. Rows past the request's end (and rows of a bad page id) are never loaded: zero bytes, zero scale.
// The loads of tile t + 1 and the page ids of tile t + 2 are in flight while tile t is converted.
// ---------------------------------------------------------------------------------------------------------------
struct H16Raw {
  uint4 w[2];
  uint32_t sf[2];
  uint2 rope;
};
__device__ __forceinline__ void h16_convert_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, int cg) {
  const int lane = ptx::lane_id();
  const int w = (threadIdx.x >> 5) - 8, hf = w >> 2, hh = lane & 1;
  const int r[3] = {lane >> 1, 16 + (lane >> 1), 4 * w + (lane >> 3)};  // two latent rows, one rope row
  const int ps_mask = (1 << P.page_shift) - 1;
  const uint32_t peer = uint32_t(cg ^ 1);
  for (int si = 0; si < n_segs; ++si) {
    const Seg seg = s.segs[si];
    const int nt = h16_tiles(seg);
    if (nt <= 0) continue;
    const int* pt = P.page_table + (long long)seg.b * P.pt_stride;
    const int tok_base = seg.tok0 + kH16Own * cg;
    auto fetch_ids = [&](int t, int (&page)[3]) {
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int tok = tok_base + t * kH16Tile + r[i];
        page[i] = tok < seg.tok_end ? pt[tok >> P.page_shift] : -1;
      }
    };
    auto fetch_rows = [&](int t, const int (&page)[3], H16Raw& R) {
      long long row[3];
      bool live[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int tok = tok_base + t * kH16Tile + r[i];
        live[i] = tok < seg.tok_end;
        // a stale or corrupt id is never dereferenced: the row reads as zeros and the call is flagged
        if (live[i] && uint32_t(page[i]) >= uint32_t(P.num_pages)) atomicExch(P.header, int(kBadPage)), live[i] = false;
        row[i] = ((long long)page[i] << P.page_shift) + (tok & ps_mask);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        R.w[u] = make_uint4(0, 0, 0, 0), R.sf[u] = 0;
        if (live[u]) {
          R.w[u] = __ldg(reinterpret_cast<const uint4*>(P.ckv + row[u] * 256 + 32 * w + 16 * hh));
          R.sf[u] = __ldg(reinterpret_cast<const unsigned short*>(P.sf + row[u] * 32 + 4 * w + 2 * hh));
        }
      }
      R.rope = make_uint2(0, 0);
      if (live[2]) R.rope = __ldg(reinterpret_cast<const uint2*>(P.kpe + row[2] * 64 + 8 * (lane & 7)));
    };
    int page[3];
    H16Raw raw;
    fetch_ids(0, page);
    fetch_rows(0, page, raw);
    fetch_ids(1, page);
    for (int t = 0; t < nt; ++t, ++it) {
      const uint32_t kb = it & 1;
      uint4 o[2][4], orope;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t s2 = ptx::e4m3x2_to_f16x2(uint16_t(raw.sf[u]));  // scales of the unit's two blocks
        const uint32_t sc[2] = {__byte_perm(s2, s2, 0x1010), __byte_perm(s2, s2, 0x3232)};
        const uint32_t words[4] = {raw.w[u].x, raw.w[u].y, raw.w[u].z, raw.w[u].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t e[4];
          ptx::e2m1x8_to_f16x8(words[c], e);
          o[u][c] = make_uint4(ptx::hmul2(e[0], sc[c >> 1]), ptx::hmul2(e[1], sc[c >> 1]), ptx::hmul2(e[2], sc[c >> 1]), ptx::hmul2(e[3], sc[c >> 1]));
        }
      }
      orope = make_uint4(ptx::e4m3x2_to_f16x2(uint16_t(raw.rope.x)), ptx::e4m3x2_to_f16x2(uint16_t(raw.rope.x >> 16)),
                         ptx::e4m3x2_to_f16x2(uint16_t(raw.rope.y)), ptx::e4m3x2_to_f16x2(uint16_t(raw.rope.y >> 16)));
      if (t + 1 < nt) fetch_rows(t + 1, page, raw);
      if (t + 2 < nt) fetch_ids(t + 2, page);
      // the panel is part B of CTA hf (released by its PV) and part A of the other one (released by its QK^T); the rope
      // panel is part A of both
      if (it >= 2) {
        const uint32_t ph = ((it >> 1) - 1) & 1;
        bool ok = ptx::mbar_wait(&s.free_a[hf ^ 1][kb], ph, &s.abort_flag) && ptx::mbar_wait(&s.free_a[hf][kb], ph, &s.abort_flag);
        ok = ok && ptx::mbar_wait(&s.free_b[hf][kb], ph, &s.abort_flag);
        if (!__all_sync(~0u, ok)) return;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint8_t* out_row = s.kv[kb][w] + (kH16Own * cg + r[u]) * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) *reinterpret_cast<uint4*>(out_row + (uint32_t((4 * hh + c) ^ (r[u] & 7)) << 4)) = o[u][c];
      }
      *reinterpret_cast<uint4*>(s.kv[kb][8] + (kH16Own * cg + r[2]) * 128 + (uint32_t((lane & 7) ^ (r[2] & 7)) << 4)) = orope;
      ptx::fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        // the peer's tile gets the same bytes; they complete on its barrier of the part they belong to
        const uint8_t* src = s.kv[kb][w] + kH16Own * cg * 128;
        const uint8_t* rsrc = s.kv[kb][8] + (kH16Own * cg + 4 * w) * 128;
        uint64_t* peer_full = uint32_t(hf) == peer ? &s.full_b[kb] : &s.full_a[kb];
        ptx::bulk_copy_to_cta(ptx::map_to_cta(src, peer), src, 4096, ptx::map_to_cta(peer_full, peer));
        ptx::bulk_copy_to_cta(ptx::map_to_cta(rsrc, peer), rsrc, 512, ptx::map_to_cta(&s.full_a[kb], peer));
        if (w == 0) ptx::mbar_arrive_expect_tx(&s.full_a[kb], kH16PeerA);  // what the peer will send for this tile
        else ptx::mbar_arrive(&s.full_a[kb]);
        if (hf == cg) {
          if ((w & 3) == 0) ptx::mbar_arrive_expect_tx(&s.full_b[kb], kH16PeerB);
          else ptx::mbar_arrive(&s.full_b[kb]);
        }
        if (w == 0) s.progress = it + 1;
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// roles: MMA issue
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void h16_qk_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, uint32_t& seg_count, int cg) {
  const bool leader = ptx::elect_one();
  const uint32_t tm = s.tmem_base;
  const uint32_t idesc = ptx::instr_desc(kH16Rows, kH16Tile, ptx::FMT_F16, ptx::FMT_F16, false, false);
  const uint64_t q_desc = ptx::smem_desc_sw128(ptx::smem_u32(s.q[0]), 16, 1024);
  for (int si = 0; si < n_segs; ++si) {
    const int nt = h16_tiles(s.segs[si]);
    if (nt <= 0) continue;
    if (!__all_sync(~0u, ptx::mbar_wait(&s.q_full, seg_count & 1, &s.abort_flag))) return;
    ++seg_count;
    for (int t = 0; t < nt; ++t, ++it) {
      const uint32_t kb = it & 1;
      const uint64_t k_desc = ptx::smem_desc_sw128(ptx::smem_u32(s.kv[kb][0]), 16, 1024);
      // the four latent panels of one half: channels [0, 256) have Q in tensor memory, [256, 512) in shared memory
      auto half = [&](int h, uint32_t accum) {
        if (h == 0) {
#pragma unroll 1
          for (int k = 0; k < 16; ++k)
            ptx::mma_f16_ts(tm + H16Cols::S, tm + H16Cols::QN + 8 * k, k_desc + (((k >> 2) * kH16Panel + (k & 3) * 32) >> 4), idesc, accum | k);
        } else {
#pragma unroll 1
          for (int k = 0; k < 16; ++k)
            ptx::mma_f16_ss(tm + H16Cols::S, q_desc + (((k >> 2) * (kH16Rows * 128) + (k & 3) * 32) >> 4),
                            k_desc + (((4 + (k >> 2)) * kH16Panel + (k & 3) * 32) >> 4), idesc, accum | k);
        }
      };
      // the softmax warps have read the scores of tile it - 1; part A of this tile is in place
      if (!__all_sync(~0u, it < 1 || ptx::mbar_wait(&s.s_free, (it - 1) & 1, &s.abort_flag))) return;
      if (!__all_sync(~0u, ptx::mbar_wait(&s.full_a[kb], (it >> 1) & 1, &s.abort_flag))) return;
      ptx::tc_fence_after_sync();
      if (leader) {
        half(cg ^ 1, 0);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          ptx::mma_f16_ts(tm + H16Cols::S, tm + H16Cols::QR + 8 * ks, k_desc + ((8 * kH16Panel + ks * 32) >> 4), idesc, 1);
        ptx::mma_commit_pair(&s.free_a[cg][kb]);
      }
      __syncwarp();
      if (!__all_sync(~0u, ptx::mbar_wait(&s.full_b[kb], (it >> 1) & 1, &s.abort_flag))) return;
      ptx::tc_fence_after_sync();
      if (leader) {
        half(cg, 1);
        ptx::mma_commit(&s.s_full);
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ void h16_pv_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, int cg) {
  const bool leader = ptx::elect_one();
  const uint32_t tm = s.tmem_base;
  // B = V read MN-major: N = 256 channels = four 128-byte runs (panels 4 cg .. 4 cg + 3), K = 16 token rows
  const uint32_t idesc = ptx::instr_desc(kH16Rows, 256, ptx::FMT_F16, ptx::FMT_F16, false, true);
  for (int si = 0; si < n_segs; ++si) {
    const int nt = h16_tiles(s.segs[si]);
    for (int t = 0; t < nt; ++t, ++it) {
      const uint32_t kb = it & 1;
      if (!__all_sync(~0u, ptx::mbar_wait(&s.p_full, it & 1, &s.abort_flag))) return;
      ptx::tc_fence_after_sync();
      if (leader) {
        const uint64_t v_desc = ptx::smem_desc_sw128(ptx::smem_u32(s.kv[kb][4 * cg]), kH16Panel, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          ptx::mma_f16_ts(tm + H16Cols::O, tm + H16Cols::P + 8 * ks, v_desc + ((ks * 16 * 128) >> 4), idesc, (t | ks) != 0);
        ptx::mma_commit(&s.pv_done);
        ptx::mma_commit_pair(&s.free_b[cg][kb]);
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------------------------------------------
// role: softmax + query load + epilogue (8 warps). Warp w: tensor-memory quadrant w % 4 (query rows 32 (w % 4) .. + 31),
// half w / 4: the two warps of a quadrant share each row's tile (32 tokens each), its O row (128 columns each) and its
// query (latent channels [256 half, +256); the upper half also takes the rope part). A row's running max must be the
// same in both, so the pair votes at a named barrier once per tile and, only when some row outgrows its max by 2^8,
// exchanges the maxima through shared memory. A quadrant without live rows only keeps the barriers going.
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void h16_softmax_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, int cg) {
  const int lane = ptx::lane_id(), warp = threadIdx.x >> 5;
  const int quad = warp & 3, half = warp >> 2;
  const int h = quad * 32 + lane;  // row of the group = tensor-memory lane
  const uint32_t tm_lane = s.tmem_base + (uint32_t(quad * 32) << 16);
  const uint32_t pair_bar = 1 + quad;
  constexpr float kGrow = 8.f;
  for (int si = 0; si < n_segs; ++si) {
    const Seg seg = s.segs[si];
    const int nt = h16_tiles(seg);
    if (nt <= 0) continue;
    const int r0 = seg.hg * P.heads_per_cta;
    const int live_rows = P.heads - r0 < P.heads_per_cta ? P.heads - r0 : P.heads_per_cta;
    if (quad * 32 >= live_rows) {
      if (lane == 0) ptx::mbar_arrive(&s.q_full);
      for (int t = 0; t < nt; ++t, ++it) {
        if (!__all_sync(~0u, ptx::mbar_wait(&s.s_full, it & 1, &s.abort_flag))) return;
        if (lane == 0) ptx::mbar_arrive(&s.s_free);
        // (not into the phase of the tile before: its P is complete once its PV is)
        if (!__all_sync(~0u, it < 1 || ptx::mbar_wait(&s.pv_done, (it - 1) & 1, &s.abort_flag))) return;
        if (lane == 0) ptx::mbar_arrive(&s.p_full);
        __syncwarp();
      }
      continue;
    }
    // ---- query: every MMA that read the previous segment's query has completed (the scores of its last tile were consumed)
    const int hq = h < live_rows ? h : live_rows - 1;  // a dead row of a live quadrant repeats the last one; it is not written out
    const long long row = (long long)seg.b * P.heads + r0 + hq;
    const uint4* qn = reinterpret_cast<const uint4*>(P.q_nope + row * CKV) + 32 * half;
    const uint4* qp = reinterpret_cast<const uint4*>(P.q_pe + row * KPE);
    const float ratio = P.kpe_scale / P.ckv_scale;  // rope scores in units of the latent ones
#pragma unroll
    for (int l = 0; l < 4; ++l) ptx::prefetch_l2(reinterpret_cast<const char*>(qn) + 128 * l);
    if (half) ptx::prefetch_l2(qp);
    // largest magnitude, as BF16 bits (ordered like integers); an infinity or NaN shows as >= 0x7F80
    auto amax_bits = [](const uint4* src, int n) {
      uint32_t m2 = 0;
#pragma unroll 1
      for (int c0 = 0; c0 < n; c0 += 8) {
        uint4 v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = __ldg(src + c0 + c);
#pragma unroll
        for (int c = 0; c < 8; ++c)
          m2 = ptx::max_s16x2(ptx::max_s16x2(m2, ptx::max_s16x2(v[c].x & 0x7FFF7FFFu, v[c].y & 0x7FFF7FFFu)),
                              ptx::max_s16x2(v[c].z & 0x7FFF7FFFu, v[c].w & 0x7FFF7FFFu));
      }
      return max(m2 & 0xFFFFu, m2 >> 16);
    };
    // non-finite elements become 0: they have no meaningful result anyway, the rest of the row stays intact
    auto clean = [](uint32_t x) {
      if ((x & 0x7F80u) == 0x7F80u) x &= 0xFFFF0000u;
      if ((x & 0x7F800000u) == 0x7F800000u) x &= 0x0000FFFFu;
      return x;
    };
    uint32_t bits = amax_bits(qn, 32), bits_p = half ? amax_bits(qp, KPE / 8) : 0u;
    const bool odd = bits >= 0x7F80u || bits_p >= 0x7F80u;
    if (odd) {  // once more, without the non-finite ones
      bits = bits_p = 0;
      auto fold = [&](const uint4& v, uint32_t m) {
        const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t c = clean(wv[j]) & 0x7FFF7FFFu;
          m = max(m, max(c & 0xFFFFu, c >> 16));
        }
        return m;
      };
#pragma unroll 1
      for (int c = 0; c < 32; ++c) bits = fold(qn[c], bits);
      if (half)
#pragma unroll 1
        for (int c = 0; c < KPE / 8; ++c) bits_p = fold(qp[c], bits_p);
    }
    s.xch[half][h] = fmaxf(__uint_as_float(bits << 16), __uint_as_float(bits_p << 16) * ratio);
    ptx::bar_sync(pair_bar, 64);
    // the row is scaled by 2^(14 - e), e = floor(log2(row maximum)): FP16 then holds a BF16 element exactly down to 2^-29 of
    // the maximum. The sign of the softmax scale goes into Q, so that a larger accumulator is always a larger score.
    int e = int(__float_as_uint(fmaxf(s.xch[0][h], s.xch[1][h])) >> 23) - 127;
    e = e < -80 ? -80 : e > 126 ? 126 : e;
    float up = __uint_as_float(uint32_t(14 - e + 127) << 23);
    const float qa = fmaxf(fabsf(P.sm_scale_log2) * P.ckv_scale * __uint_as_float(uint32_t(e - 14 + 127) << 23), 1e-37f);
    up = P.sm_scale_log2 < 0.f ? -up : up;
    auto f16x8 = [&](uint4 v, float sc) {
      if (odd) v = make_uint4(clean(v.x), clean(v.y), clean(v.z), clean(v.w));
      auto two = [&](uint32_t x) { return ptx::f32x2_to_f16x2(__uint_as_float(x << 16) * sc, __uint_as_float(x & 0xFFFF0000u) * sc); };
      return make_uint4(two(v.x), two(v.y), two(v.z), two(v.w));
    };
#pragma unroll 1
    for (int c0 = 0; c0 < 32; c0 += 8) {  // 64 channels per trip
      uint4 v[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = __ldg(qn + c0 + c);
#pragma unroll
      for (int c = 0; c < 8; ++c) v[c] = f16x8(v[c], up);
      if (half == 0) {
        uint32_t col[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) col[4 * c] = v[c].x, col[4 * c + 1] = v[c].y, col[4 * c + 2] = v[c].z, col[4 * c + 3] = v[c].w;
        ptx::tmem_st32(tm_lane + H16Cols::QN + 4 * c0, col);
      } else {
        uint8_t* dst = s.q[c0 >> 3] + h * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(dst + (uint32_t(c ^ (h & 7)) << 4)) = v[c];
      }
    }
    if (half) {
      uint32_t col[32];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4 v = __ldg(qp + c);
        if (odd) v = make_uint4(clean(v.x), clean(v.y), clean(v.z), clean(v.w));
        const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
          col[4 * c + j] = ptx::f32x2_to_f16x2(__uint_as_float(wv[j] << 16) * ratio * up, __uint_as_float(wv[j] & 0xFFFF0000u) * ratio * up);
      }
      ptx::tmem_st32(tm_lane + H16Cols::QR, col);
      ptx::fence_proxy_async_smem();
    }
    ptx::tmem_wait_st();
    ptx::tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&s.q_full);

    float m = -INFINITY, l = 0.f;  // m is identical in the row's two threads; l is this thread's share of the sum
    for (int t = 0; t < nt; ++t, ++it) {
      const bool ok = ptx::mbar_wait(&s.s_full, it & 1, &s.abort_flag);
      ptx::tc_fence_after_sync();
      const int nvalid = seg.tok_end - (seg.tok0 + t * kH16Tile) - 32 * half;  // this warp's columns at or beyond it are masked
      uint32_t sr[32];
      if (ok) {
        ptx::tmem_ld32(tm_lane + H16Cols::S + 32 * half, sr);
        ptx::tmem_wait_ld();
      }
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&s.s_free);  // QK^T of tile it + 1 may overwrite the scores
      if (!ok || nvalid < 32) {
#pragma unroll
        for (int j = 0; j < 32; ++j) sr[j] = (ok && j < nvalid) ? sr[j] : 0xFF800000u;
      }
      float mxs[4] = {__uint_as_float(sr[0]), __uint_as_float(sr[1]), __uint_as_float(sr[2]), __uint_as_float(sr[3])};
#pragma unroll
      for (int j = 4; j + 8 <= 32; j += 8)  // four chains of three-input maxima
#pragma unroll
        for (int k = 0; k < 4; ++k) mxs[k] = ptx::max3(mxs[k], __uint_as_float(sr[j + 2 * k]), __uint_as_float(sr[j + 2 * k + 1]));
#pragma unroll
      for (int k = 0; k < 4; ++k) mxs[k] = fmaxf(mxs[k], __uint_as_float(sr[28 + k]));
      const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * qa;
      if (ptx::bar_red_or(pair_bar, 64, !ok || mx > m + kGrow)) {
        s.xch[half][h] = mx;
        if (ptx::bar_red_or(pair_bar, 64, s.abort_flag != 0)) return;  // uniform in the pair, whoever raised the flag
        const float mxp = fmaxf(s.xch[0][h], s.xch[1][h]);
        const bool need = mxp > m + kGrow;
        const float mn = need ? mxp : m;
        const float corr = need ? ((m == -INFINITY) ? 0.f : ptx::ex2(m - mn)) : 1.f;
        l *= corr, m = mn;
        if (t > 0) {  // O holds the segment's earlier tiles: wait for the PV of tile it - 1, then scale this thread's half row
          const bool okv = ptx::mbar_wait(&s.pv_done, (it - 1) & 1, &s.abort_flag);
          if (ptx::bar_red_or(pair_bar, 64, !okv)) return;
          ptx::tc_fence_after_sync();
#pragma unroll 1
          for (int c0 = 0; c0 < 128; c0 += 32) {
            uint32_t o[32];
            ptx::tmem_ld32(tm_lane + H16Cols::O + 128 * half + c0, o);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
            ptx::tmem_st32(tm_lane + H16Cols::O + 128 * half + c0, o);
          }
          ptx::tmem_wait_st();
        }
      }
      // P = 2^(s qa - m) as FP16 into this warp's 16 of the tile's 32 P columns, once PV of tile it - 1 has read them
      const float neg_m = (m == -INFINITY) ? 0.f : -m;
      uint32_t pk[16];
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const float p0 = ptx::ex2(fmaf(__uint_as_float(sr[2 * c]), qa, neg_m)), p1 = ptx::ex2(fmaf(__uint_as_float(sr[2 * c + 1]), qa, neg_m));
        ls[c & 3] += p0 + p1;
        pk[c] = ptx::f32x2_to_f16x2(p0, p1);
      }
      l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
      if (it >= 1) {  // (a wait that gives up raises the abort flag; the next vote or the epilogue ends the role for both warps)
        ptx::mbar_wait(&s.pv_done, (it - 1) & 1, &s.abort_flag);
        ptx::tc_fence_after_sync();
      }
      ptx::tmem_st16(tm_lane + H16Cols::P + 16 * half, pk);
      ptx::tmem_wait_st();
      ptx::tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(&s.p_full);
    }

    // ---- segment epilogue: wait for the last PV, add the two halves of the sum, write this thread's 128 of the row's 256
    // channels of the normalised partial
    const bool ok = ptx::mbar_wait(&s.pv_done, (it - 1) & 1, &s.abort_flag);
    s.xl[half][h] = l;
    if (ptx::bar_red_or(pair_bar, 64, !ok)) return;
    ptx::tc_fence_after_sync();
    const float lt = s.xl[0][h] + s.xl[1][h];
    const float inv = lt > 0.f ? P.ckv_scale / lt : 0.f;
    const long long slot = (long long)seg.cta + seg.w;
    float* orow = P.o_part + (slot * P.heads_per_cta + h) * CKV + 256 * cg + 128 * half;
#pragma unroll 1
    for (int c0 = 0; c0 < 128; c0 += 32) {
      uint32_t o[32];
      ptx::tmem_ld32(tm_lane + H16Cols::O + 128 * half + c0, o);
      ptx::tmem_wait_ld();
      if (h < live_rows) {
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          *reinterpret_cast<float4*>(orow + c0 + j) = make_float4(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv,
                                                                  __uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv);
      }
    }
    if (cg == 0 && half == 0 && h < live_rows) P.lse_part[slot * P.heads_per_cta + h] = lt > 0.f ? m + log2f(lt) : -INFINITY;
    ptx::tc_fence_before_sync();
    ptx::bar_sync(pair_bar, 64);  // s.xl and s.xch are reused by the next segment
  }
}

// ---------------------------------------------------------------------------------------------------------------
// kernel
// ---------------------------------------------------------------------------------------------------------------
enum H16Role { kH16Softmax, kH16Convert, kH16Qk, kH16Prefetch, kH16Pv, kH16Idle };

template <int ROLE>
__device__ __forceinline__ void h16_run_role(H16Smem& s, const DecodeParams& P) {
  const int pair = blockIdx.x >> 1, cg = blockIdx.x & 1;
  const int2 range = P.cta_range[pair];
  uint32_t it = 0, seg_count = 0;  // every role advances its own copies identically
  for (int w0 = range.x; w0 < range.y; w0 += kSegBatch) {
    const int n_segs = range.y - w0 < kSegBatch ? range.y - w0 : kSegBatch;
    if (ROLE == kH16Softmax && int(threadIdx.x) < n_segs) {
      Seg g = P.segs[(long long)pair + w0 + threadIdx.x];
      if (g.cta != pair || g.w != w0 + int(threadIdx.x)) g.ntiles = 0;  // empty item or foreign slot
      s.segs[threadIdx.x] = g;
    }
    __syncthreads();
    if (ROLE == kH16Softmax) h16_softmax_role(s, P, n_segs, it, cg);
    if (ROLE == kH16Convert) h16_convert_role(s, P, n_segs, it, cg);
    if (ROLE == kH16Qk) h16_qk_role(s, P, n_segs, it, seg_count, cg);
    if (ROLE == kH16Prefetch) h16_prefetch_role(s, P, n_segs, it, cg);
    if (ROLE == kH16Pv) h16_pv_role(s, P, n_segs, it, cg);
    __syncthreads();
    if (s.abort_flag) break;
  }
  // The releases of the last two tiles come from the peer as well: see them arrive before this CTA's memory goes away. (The
  // convert warps have seen those of all earlier tiles, so each barrier is at most one phase short.)
  if (ROLE == kH16Prefetch && !s.abort_flag)
    for (uint32_t j = it >= 2 ? it - 2 : 0; j < it; ++j)
      for (int x = 0; x < 2; ++x)
        ptx::mbar_wait(&s.free_a[x][j & 1], (j >> 1) & 1, &s.abort_flag), ptx::mbar_wait(&s.free_b[x][j & 1], (j >> 1) & 1, &s.abort_flag);
}

__global__ void __launch_bounds__(kH16Threads, 1) mla_decode_hm16_kernel(const DecodeParams P) {
  extern __shared__ uint8_t smem_raw[];
  H16Smem& s = *reinterpret_cast<H16Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&s.full_a[i], 8), ptx::mbar_init(&s.full_b[i], 4);
      for (int x = 0; x < 2; ++x) ptx::mbar_init(&s.free_a[x][i], 1), ptx::mbar_init(&s.free_b[x][i], 1);
    }
    ptx::mbar_init(&s.s_full, 1), ptx::mbar_init(&s.s_free, 8);
    ptx::mbar_init(&s.p_full, 8), ptx::mbar_init(&s.pv_done, 1);
    ptx::mbar_init(&s.q_full, 8);
    s.abort_flag = 0, s.progress = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 16) {
    ptx::tmem_alloc(&s.tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  ptx::cluster_sync();  // both CTAs' barriers are initialised before either signals the other's
  ptx::tc_fence_after_sync();
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();  // after the wait: the combine kernel reads a schedule kernel's output as soon as it starts
  // the query panels are written by this CTA's own softmax warps only (the peer writes to kv): free until then
  if (P.inline_sched) publish_own_schedule<kH16Threads>(reinterpret_cast<int*>(s.q[0]), P, blockIdx.x >> 1);

  // register budgets, warp group by warp group; the pool is the launch allocation, 20 warps x 96
  constexpr int kLaunchRegs = 96, kSoftmaxRegs = 104, kConvertRegs = 112, kIssueRegs = 48;
  static_assert(8 * kSoftmaxRegs + 8 * kConvertRegs + 4 * kIssueRegs <= 20 * kLaunchRegs, "register budgets exceed the CTA's allocation");
  if (warp < 8) {
    ptx::reg_alloc<kSoftmaxRegs>();
    h16_run_role<kH16Softmax>(s, P);
  } else if (warp < 16) {
    ptx::reg_alloc<kConvertRegs>();
    h16_run_role<kH16Convert>(s, P);
  } else {
    ptx::reg_dealloc<kIssueRegs>();
    if (warp == 16) h16_run_role<kH16Qk>(s, P);
    else if (warp == 17) h16_run_role<kH16Prefetch>(s, P);
    else if (warp == 18) h16_run_role<kH16Pv>(s, P);
    else h16_run_role<kH16Idle>(s, P);
  }

  ptx::tc_fence_before_sync();
  ptx::cluster_sync();  // neither CTA leaves while the other may still write to its shared memory or signal its barriers
  if (warp == 16) ptx::tmem_dealloc(s.tmem_base, kTmemCols);
  if (threadIdx.x == 0 && s.abort_flag) atomicExch(P.header, int(kWaitTimeout));
}

}  // namespace mla
