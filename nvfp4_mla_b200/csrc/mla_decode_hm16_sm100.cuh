// Weight-absorbed MLA decode for many query rows per request (heads, or heads x query tokens), 16-bit mode, with the query
// rows as the M dimension of both MMAs. The 16-head kernel (mla_decode_vt_sm100.cuh) converts a token once per 16 heads; here one FP16 copy of a
// token serves up to 128 rows:
//
//   HBM --L2 prefetch, 16-byte loads--> convert warps' registers --> K/V tile in smem, FP16, [token][channel], 128-byte swizzle
//   QK^T : S[row, token] = Q[row, 576] . K^T    A = Q (FP16) from tensor memory (latent 0..255, rope) / smem (latent 256..511),
//                                               B = the K/V tile read K-major, N = 64 tokens
//   PV   : O[row, chan] += P[row, token] . V    A = P (FP16) from tensor memory, written there by the softmax threads,
//                                               B = the same K/V tile read MN-major, N = 256 channels, K = 16 tokens
// Both K and V are exact in FP16 (e2m1 x e4m3 has six significant bits). The latent part of Q (a BF16 has eight) is
// held times a power of two per row: exact, but for elements so small that they are off by up to 2^-25 of the row's maximum. Its
// rope part is multiplied with kpe_scale / ckv_scale and rounded to FP16. The accumulators are fp32.
//
// O for 128 rows x 512 channels would need all 512 tensor-memory columns, so a PAIR of CTAs shares a request: both compute
// the full scores, CTA `cg` accumulates channels [256 cg, 256 cg + 256). The pair is one unit of the schedule and writes one
// partial slot; its CTAs do not communicate (the second read of a token is an L2 hit). An earlier form was a cluster of two
// that shared the conversion, each CTA sending half of every tile to its peer by bulk copies through distributed shared
// memory: 981 us instead of 884 (128 heads, two requests of 1M tokens; 1740 with the 16-head kernel), because a tile's first
// MMA waited for the peer's PV of two tiles before, its conversion and the transfer.
//
// What bounds it from below is the tensor pipe. Per 64-token tile and CTA 20 MMAs of 32 cycles (A in tensor memory), 16 of
// 48 (A in shared memory, bound by the operand read) and 4 of 128 for PV: 1920 cycles, of about 2700 measured. Storage
// allows two K/V tiles only (Q 144 KB, O 128 KB and S / P 48 KB of tensor memory + shared memory leave room for 2.2), so a
// tile is handed over in two parts: A = the nine panels minus this CTA's PV half (free as soon as QK^T has read them), B =
// the four panels PV reads. The next tile's part A is converted and multiplied while PV of the previous tile still holds
// part B. What limits a tile now is the softmax warps' serial chain (scores -> vote -> exponentials -> P), behind which S has
// one buffer only; long calls run at the power limit (about 1.4 GHz).
//
// Tensor memory (512 columns): Q latent 0..255: 0..127 | Q rope: 128..159 | S: 160..223 | P: 224..255 | O: 256..511.
// Warp roles (896 threads): 0-7 softmax + query load + epilogue, 8-23 dequantise (warp = 32 rows of a 64-channel panel), 24
// QK^T issue, 25 L2 prefetch, 26 PV issue. Every wait is bounded (ptx::mbar_wait).
#pragma once
#include <climits>
#include <type_traits>

#include "mla_decode_sm100.cuh"

namespace mla {

constexpr int kH16Threads = 896;
constexpr int kH16Rows = 128;              // query rows per CTA pair = MMA M (at most; the rest of M is dead)
constexpr int kH16Tile = 64;               // tokens per tile
constexpr int kH16Own = kH16Tile / 2;      // token rows of a tile that one CTA of the pair prefetches into L2
constexpr int kH16Panel = kH16Tile * 128;  // one 64-channel panel of the FP16 tile
constexpr int kH16Ahead = 6;               // tiles between a load and its L2 prefetch

struct H16Smem {
  alignas(1024) uint8_t q[4][kH16Rows * 128];   // latent channels 256..511 of Q, FP16, row = query row, four panels of 64 channels
  alignas(1024) uint8_t kv[2][9][kH16Panel];    // panels 0..7: latent channels, panel 8: rope
  Seg segs[kSegBatch];
  alignas(8) uint64_t full_a[2], full_b[2];     // part of the tile in place (eight convert warps each)
  uint64_t free_a[2], free_b[2];                // buffer part released: part A by QK^T, part B by PV
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
  // one request per run of contiguous rows (a page, or this CTA's share of the tile), by the lane of its first row
  const int run = P.page_shift >= 5 ? kH16Own : 1 << P.page_shift;
  if ((lane & (run - 1)) == 0) {
    ptx::bulk_prefetch_l2(P.ckv + row * 256, run * 256);
    ptx::bulk_prefetch_l2(P.kpe + row * 64, run * 64);
    ptx::bulk_prefetch_l2(P.sf + row * 32, run * 32);
  }
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
// role: dequantise (16 warps). Warp cw: panel cw % 8 (64 channels), rows [32 (cw / 8), +32) of the tile; a lane takes half a
// panel row (16 packed bytes = two scale blocks) of rows lane / 2 and 16 + lane / 2, so that a warp's load touches 16 lines
// and its 16-byte stores are conflict-free. The warps of part A also move the rope panel (8 rows each, eight lanes per row).
// The cache row of a token is looked up by one lane and handed round by shuffle. Rows past the request's end and rows of a
// bad page id are never loaded: zero bytes, zero scale. With several query tokens per request the last tokens are not seen by
// every row, and a row that masks a token multiplies its value with probability 0, so a NaN block scale must not reach that value:
// there the block becomes 0, and the token's rope part, which only enters scores, NaN. The loads of tile t + 1 are issued as soon as tile t's bytes have
// been converted, the page ids of tile t + 2 behind them.
// ---------------------------------------------------------------------------------------------------------------
template <bool part_a>  // whether the warp's panel belongs to part A
__device__ __forceinline__ void h16_convert_warps(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it) {
  const int lane = ptx::lane_id();
  const int cw = (threadIdx.x >> 5) - 8, w = cw & 7, v = cw >> 3, hh = lane & 1;
  uint64_t* const full = part_a ? s.full_a : s.full_b;
  uint64_t* const freed = part_a ? s.free_a : s.free_b;
  const int rope_row = 8 * (w & 3) + (lane >> 3);  // of this warp's 32 rows; the lane's second one is 4 rows further
  // per-lane byte offsets: latent chunk c of a row r is at 16 ((4 hh + c) ^ (r % 8)), and r % 8 is the same for both rows
  const uint32_t kv0 = ptx::smem_u32(s.kv[0][0]);
  const uint32_t dst0 = kv0 + w * kH16Panel + (32 * v + (lane >> 1)) * 128 + ((uint32_t(4 * hh) ^ uint32_t((lane >> 1) & 4)) << 4);
  const uint32_t swz = uint32_t((lane >> 1) & 3) << 4;
  const uint32_t rope0 = kv0 + 8 * kH16Panel + (32 * v + rope_row) * 128, rope_c = uint32_t(lane & 7), rope_s = uint32_t(rope_row & 7);
  const uint8_t* const ckv0 = P.ckv + 32 * w + 16 * hh;
  const uint8_t* const sf0 = P.sf + 4 * w + 2 * hh;
  const uint8_t* const kpe0 = P.kpe + 8 * (lane & 7);
  auto has_nan = [](uint32_t w) { return __vcmpeq4(w & 0x7F7F7F7Fu, 0x7F7F7F7Fu) != 0u; };
  for (int si = 0; si < n_segs; ++si) {
    const Seg seg = s.segs[si];
    const int nt = h16_tiles(seg);
    if (nt <= 0) continue;
    const int* pt = P.page_table + (long long)seg.b * P.pt_stride;
    const int first_masked = P.q_len > 1 ? P.kv_lens[seg.b] - (P.q_len - 1) : INT_MAX;  // first token that some row does not see
    uint4 rw[2];
    uint32_t rs[2];
    uint2 rr[2];
    int ru[2], rj[2] = {0, 0};           // cache rows of the two latent units and the two rope chunks, negative: none
    int tok = seg.tok0 + 32 * v + lane;  // this lane's token of the tile being fetched
    // No load sits behind a branch (it would be waited for where the branches meet, one trip to memory per load instead of
    // one per tile): tokens past the end look up the last live token's page, dead rows read cache row 0 and are zeroed where
    // their bytes are used, and the fetches past the last tile are issued like the others.
    auto fetch_id = [&](int tk) { return __ldg(pt + ((tk < seg.tok_end ? tk : seg.tok_end - 1) >> P.page_shift)); };
    auto fetch_rows = [&](int page) {
      const bool live = tok < seg.tok_end, good = uint32_t(page) < uint32_t(P.num_pages);
      // a stale or corrupt id is never dereferenced: the row reads as zeros and the call is flagged
      if (live && !good) atomicExch(P.header, int(kBadPage));
      const int row = live && good ? (page << P.page_shift) + (tok & ((1 << P.page_shift) - 1)) : -1;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        ru[u] = __shfl_sync(~0u, row, 16 * u + (lane >> 1));
        const long long at = ru[u] < 0 ? 0 : ru[u];
        rw[u] = __ldg(reinterpret_cast<const uint4*>(ckv0 + at * 256));
        rs[u] = __ldg(reinterpret_cast<const unsigned short*>(sf0 + at * 32));
      }
      if constexpr (part_a) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          rj[j] = __shfl_sync(~0u, row, rope_row + 4 * j);
          rr[j] = __ldg(reinterpret_cast<const uint2*>(kpe0 + (long long)(rj[j] < 0 ? 0 : rj[j]) * 64));
        }
      }
      tok += kH16Tile;
    };
    // the tile in the registers, into buffer `buf`; MASKED: rows from `first` on hold tokens that some query row does not see
    auto convert = [&](auto masked, uint32_t buf, int first) {
      constexpr bool MASKED = decltype(masked)::value;
      if constexpr (MASKED) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (16 * u + (lane >> 1) < first) continue;
          if ((rs[u] & 0x7Fu) == 0x7Fu) rs[u] &= 0xFF00u;
          if ((rs[u] & 0x7F00u) == 0x7F00u) rs[u] &= 0x00FFu;
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint32_t s2 = ru[u] < 0 ? 0u : ptx::e4m3x2_to_f16x2(uint16_t(rs[u]));  // scales of the unit's two blocks
        const uint32_t sc[2] = {__byte_perm(s2, s2, 0x1010), __byte_perm(s2, s2, 0x3232)};
        const uint32_t words[4] = {rw[u].x, rw[u].y, rw[u].z, rw[u].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t e[4];
          ptx::e2m1x8_to_f16x8(words[c], e);
          ptx::sts128(dst0 + buf + u * 2048 + ((uint32_t(c) << 4) ^ swz), ptx::hmul2(e[0], sc[c >> 1]), ptx::hmul2(e[1], sc[c >> 1]),
                      ptx::hmul2(e[2], sc[c >> 1]), ptx::hmul2(e[3], sc[c >> 1]));
        }
      }
      if constexpr (part_a) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          uint2 x = rj[j] < 0 ? make_uint2(0, 0) : rr[j];
          if constexpr (MASKED) {
            if (rj[j] >= 0 && rope_row + 4 * j >= first) {
              const uint4* sf = reinterpret_cast<const uint4*>(P.sf + (long long)rj[j] * 32);
              const uint4 a = sf[0], b = sf[1];
              if (has_nan(a.x) || has_nan(a.y) || has_nan(a.z) || has_nan(a.w) || has_nan(b.x) || has_nan(b.y) || has_nan(b.z) || has_nan(b.w))
                x = make_uint2(0x7F7F7F7Fu, 0x7F7F7F7Fu);
            }
          }
          ptx::sts128(rope0 + buf + j * 512 + ((rope_c ^ (rope_s + 4 * j)) << 4), ptx::e4m3x2_to_f16x2(uint16_t(x.x)),
                      ptx::e4m3x2_to_f16x2(uint16_t(x.x >> 16)), ptx::e4m3x2_to_f16x2(uint16_t(x.y)), ptx::e4m3x2_to_f16x2(uint16_t(x.y >> 16)));
        }
      }
    };
    fetch_rows(fetch_id(tok));
    int page = fetch_id(tok);
    for (int t = 0; t < nt; ++t, ++it) {
      const uint32_t kb = it & 1, buf = kb * uint32_t(sizeof(s.kv[0]));
      // this part of the buffer was released by the MMAs of tile it - 2
      if (it >= 2 && !__all_sync(~0u, ptx::mbar_wait(&freed[kb], ((it >> 1) - 1) & 1, &s.abort_flag))) return;
      // a tile whose tokens every row sees (all but a request's last one, and that too with one query token) goes without the checks
      const int tok0 = tok - kH16Tile - lane;  // token of this warp's first row
      if (tok0 + 32 <= first_masked) convert(std::false_type(), buf, 0);
      else convert(std::true_type(), buf, first_masked - tok0);
      ptx::fence_proxy_async_smem();
      __syncwarp();
      ptx::mbar_arrive_if(&full[kb], lane == 0);
      if (cw == 0 && lane == 0) s.progress = it + 1;
      const int pg = page;
      page = fetch_id(tok + kH16Tile);
      fetch_rows(pg);
    }
  }
}

__device__ __forceinline__ void h16_convert_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, int cg) {
  if (int(((threadIdx.x >> 5) - 8) >> 2 & 1) != cg) h16_convert_warps<true>(s, P, n_segs, it);
  else h16_convert_warps<false>(s, P, n_segs, it);
}

// ---------------------------------------------------------------------------------------------------------------
// roles: MMA issue, by one elected thread behind a branch (an earlier form, every thread running the issue code with the MMAs
// predicated on the elected one, gave wrong results where the warp happened to run it diverged, and was not faster: 64 heads, 32
// ragged requests 147.5 us, this form 145.6)
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void h16_qk_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, uint32_t& seg_count, int cg) {
  const bool leader = ptx::elect_one();
  const uint32_t tm = 0;  // all 512 columns are allocated: they start at column 0 (a constant keeps the MMA operands uniform)
  const uint32_t idesc = ptx::instr_desc(kH16Rows, kH16Tile, ptx::FMT_F16, ptx::FMT_F16, false, false);
  const uint64_t q_desc = ptx::smem_desc_sw128(ptx::smem_u32(s.q[0]), 16, 1024), kv_desc = ptx::smem_desc_sw128(ptx::smem_u32(s.kv[0][0]), 16, 1024);
  const uint32_t hi = uint32_t(q_desc >> 32);
  for (int si = 0; si < n_segs; ++si) {
    const int nt = h16_tiles(s.segs[si]);
    if (nt <= 0) continue;
    if (!__all_sync(~0u, ptx::mbar_wait(&s.q_full, seg_count & 1, &s.abort_flag))) return;
    ++seg_count;
    for (int t = 0; t < nt; ++t, ++it) {
      const uint32_t kb = it & 1;
      const uint32_t k_lo = uint32_t(kv_desc) + kb * uint32_t(sizeof(s.kv[0]) >> 4);
      // the four latent panels of one half: channels [0, 256) have Q in tensor memory, [256, 512) in shared memory
      auto half = [&](int h, uint32_t accum) {
        uint32_t q = h == 0 ? tm + H16Cols::QN : uint32_t(q_desc), k = k_lo + h * (4 * kH16Panel >> 4);
        if (h == 0) {
#pragma unroll 1
          for (int p = 0; p < 4; ++p, q += 32, k += kH16Panel >> 4)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) ptx::mma_f16_ts_lo(tm + H16Cols::S, q + 8 * ks, k + 2 * ks, hi, idesc, ks ? 1u : accum | p);
        } else {
#pragma unroll 1
          for (int p = 0; p < 4; ++p, q += kH16Rows * 128 >> 4, k += kH16Panel >> 4)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) ptx::mma_f16_ss_lo(tm + H16Cols::S, q + 2 * ks, k + 2 * ks, hi, idesc, ks ? 1u : accum | p);
        }
      };
      // the softmax warps have read the scores of tile it - 1; part A of this tile is in place
      if (!__all_sync(~0u, it < 1 || ptx::mbar_wait(&s.s_free, (it - 1) & 1, &s.abort_flag))) return;
      if (!__all_sync(~0u, ptx::mbar_wait(&s.full_a[kb], (it >> 1) & 1, &s.abort_flag))) return;
      ptx::tc_fence_after_sync();
      if (leader) {
        half(cg ^ 1, 0u);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          ptx::mma_f16_ts_lo(tm + H16Cols::S, tm + H16Cols::QR + 8 * ks, k_lo + ((8 * kH16Panel + ks * 32) >> 4), hi, idesc, 1u);
        ptx::mma_commit(&s.free_a[kb]);
      }
      __syncwarp();
      if (!__all_sync(~0u, ptx::mbar_wait(&s.full_b[kb], (it >> 1) & 1, &s.abort_flag))) return;
      ptx::tc_fence_after_sync();
      if (leader) {
        half(cg, 1u);
        ptx::mma_commit(&s.s_full);
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ void h16_pv_role(H16Smem& s, const DecodeParams& P, int n_segs, uint32_t& it, int cg) {
  const bool leader = ptx::elect_one();
  const uint32_t tm = 0;  // all 512 columns are allocated: they start at column 0 (a constant keeps the MMA operands uniform)
  // B = V read MN-major: N = 256 channels = four 128-byte runs (panels 4 cg .. 4 cg + 3), K = 16 token rows
  const uint32_t idesc = ptx::instr_desc(kH16Rows, 256, ptx::FMT_F16, ptx::FMT_F16, false, true);
  for (int si = 0; si < n_segs; ++si) {
    const int nt = h16_tiles(s.segs[si]);
    for (int t = 0; t < nt; ++t, ++it) {
      const uint32_t kb = it & 1;
      if (!__all_sync(~0u, ptx::mbar_wait(&s.p_full, it & 1, &s.abort_flag))) return;
      ptx::tc_fence_after_sync();
      const uint64_t v_desc = ptx::smem_desc_sw128(ptx::smem_u32(s.kv[kb][4 * cg]), kH16Panel, 1024);
      if (leader) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          ptx::mma_f16_ts_lo(tm + H16Cols::O, tm + H16Cols::P + 8 * ks, uint32_t(v_desc) + ((ks * 16 * 128) >> 4), uint32_t(v_desc >> 32), idesc, (t | ks) != 0);
        ptx::mma_commit(&s.pv_done);
        ptx::mma_commit(&s.free_b[kb]);
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
    const int hq = h < live_rows ? h : live_rows - 1;
    // A row sees the tokens up to its own query token: token i of q_len (rows [i, i + 1) * heads / q_len of the request) stops
    // q_len - 1 - i tokens before the request's end.
    int row_end = seg.tok_end;
    if (P.q_len > 1) {
      const int i = (r0 + hq) / (P.heads / P.q_len), end = P.kv_lens[seg.b] - (P.q_len - 1 - i);
      row_end = end < row_end ? end : row_end;
    }
    // (a dead row of a live quadrant repeats the last live one and is not written out)
    const long long row = (long long)seg.b * P.heads + r0 + hq;
    const uint4* qn = reinterpret_cast<const uint4*>(P.q_nope + row * CKV) + 32 * half;
    const uint4* qp = reinterpret_cast<const uint4*>(P.q_pe + row * KPE);
    const float ratio = P.kpe_scale / P.ckv_scale;  // rope scores in units of the latent ones
#pragma unroll
    for (int l = 0; l < 4; ++l) ptx::prefetch_l2(reinterpret_cast<const char*>(qn) + 128 * l);
    if (half) ptx::prefetch_l2(qp);
    // Q as FP16 times `up`, into tensor memory / shared memory; returns the largest magnitude of the finite elements (the rope part
    // times `ratio`). Non-finite elements become 0: they have no meaningful result anyway, the rest of the row stays intact.
    auto load_query = [&](float up) {
      uint32_t m2 = 0, m2p = 0;  // BF16 magnitudes, two at a time, ordered like integers
      auto clean = [](uint32_t x) {
        if ((x & 0x7F80u) == 0x7F80u) x &= 0xFFFF0000u;
        if ((x & 0x7F800000u) == 0x7F800000u) x &= 0x0000FFFFu;
        return x;
      };
      auto two = [&](uint32_t x, float sc, uint32_t& mm) {
        x = clean(x);
        mm = ptx::max_s16x2(mm, x & 0x7FFF7FFFu);
        return ptx::f32x2_to_f16x2(__uint_as_float(x << 16) * sc, __uint_as_float(x & 0xFFFF0000u) * sc);
      };
#pragma unroll 1
      for (int c0 = 0; c0 < 32; c0 += 8) {  // 64 channels per trip
        uint4 v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = __ldg(qn + c0 + c);
        uint32_t col[32];
#pragma unroll
        for (int c = 0; c < 8; ++c)
          col[4 * c] = two(v[c].x, up, m2), col[4 * c + 1] = two(v[c].y, up, m2), col[4 * c + 2] = two(v[c].z, up, m2), col[4 * c + 3] = two(v[c].w, up, m2);
        if (half == 0) {
          ptx::tmem_st32(tm_lane + H16Cols::QN + 4 * c0, col);
        } else {
          const uint32_t dst = ptx::smem_u32(s.q[c0 >> 3]) + h * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c) ptx::sts128(dst + (uint32_t(c ^ (h & 7)) << 4), col[4 * c], col[4 * c + 1], col[4 * c + 2], col[4 * c + 3]);
        }
      }
      if (half) {
        uint32_t col[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 v = __ldg(qp + c);
          col[4 * c] = two(v.x, up * ratio, m2p), col[4 * c + 1] = two(v.y, up * ratio, m2p), col[4 * c + 2] = two(v.z, up * ratio, m2p), col[4 * c + 3] = two(v.w, up * ratio, m2p);
        }
        ptx::tmem_st32(tm_lane + H16Cols::QR, col);
      }
      return fmaxf(__uint_as_float(max(m2 << 16, m2 & 0xFFFF0000u)), __uint_as_float(max(m2p << 16, m2p & 0xFFFF0000u)) * ratio);
    };
    // The sign of the softmax scale goes into Q, so that a larger accumulator is always a larger score. The row is held times a power
    // of two, which the score's scale takes out again. Ordinary rows (maximum in [2^-8, 2^7]) are loaded in one pass, times 2^8:
    // their elements are exact from 2^-25 up and off by at most 2^-33 below, 2^-25 of the row's maximum (times 1, elements of
    // 2^-18 that meet large latent values had eight bits of error left). Any other row is loaded again times the power that puts its
    // maximum into [2^14, 2^15): exact from 2^-31 of the maximum up. The rope elements are products with `ratio`, rounded to FP16's
    // eleven bits. The tensor-memory stores are warp-wide, so the pair of warps decides together.
    constexpr int kUp = 8;
    const float sign = P.sm_scale_log2 < 0.f ? -1.f : 1.f;
    s.xch[half][h] = load_query(sign * float(1 << kUp));
    ptx::bar_sync(pair_bar, 64);
    const float amax = fmaxf(s.xch[0][h], s.xch[1][h]);
    const bool ordinary = amax >= 0x1p-8f && amax <= 0x1p7f;
    int e = -kUp;  // the row is held times 2^-e
    if (!__all_sync(~0u, ordinary)) {  // (both warps of the pair see the same maxima)
      ptx::tmem_wait_st();             // the first pass's stores go to the same columns: they have to land first
      e = int(__float_as_uint(amax) >> 23) - 127 - 14;
      e = ordinary ? -kUp : e < -94 ? -94 : e > 112 ? 112 : e;
      load_query(sign * __uint_as_float(uint32_t(127 - e) << 23));
    }
    // (never 0: a masked score is -inf and must stay so)
    const float qa = fmaxf(fabsf(P.sm_scale_log2) * P.ckv_scale * __uint_as_float(uint32_t(127 + e) << 23), 0x1p-149f);
    if (half) ptx::fence_proxy_async_smem();
    ptx::tmem_wait_st();
    ptx::tc_fence_before_sync();
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(&s.q_full);

    float m = -INFINITY, l = 0.f;  // m is identical in the row's two threads; l is this thread's share of the sum
    for (int t = 0; t < nt; ++t, ++it) {
      const bool ok = ptx::mbar_wait(&s.s_full, it & 1, &s.abort_flag);
      ptx::tc_fence_after_sync();
      const int nvalid = row_end - (seg.tok0 + t * kH16Tile) - 32 * half;  // this thread's columns at or beyond it are masked
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
      float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const float2 x = ptx::fma_f32x2(make_float2(__uint_as_float(sr[2 * c]), __uint_as_float(sr[2 * c + 1])), make_float2(qa, qa), make_float2(neg_m, neg_m));
        const float2 p = make_float2(ptx::ex2(x.x), ptx::ex2(x.y));
        ls[c & 1] = ptx::add_f32x2(ls[c & 1], p);
        pk[c] = ptx::f32x2_to_f16x2(p.x, p.y);
      }
      l += (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y);
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
    // A thread holds a row, but a store of a row per lane touches 32 lines: 32 channels at a time turn through this warp's share of
    // the quadrant's rows of s.q (the query is not needed any more), so that a store writes four rows' 128 bytes. The epilogue of
    // a CTA with one segment of 128 rows took 12000 cycles with a row per lane and takes 8000; 64 heads, 32 ragged requests: 147.5 us
    // before, 144.7 now; 128 heads, 64 requests of 300 tokens: 57.3, 54.7.
    float* const orow = P.o_part + (slot * P.heads_per_cta + 32 * quad + (lane >> 3)) * CKV + 256 * cg + 128 * half + 4 * (lane & 7);
#pragma unroll 1
    for (int c0 = 0; c0 < 128; c0 += 32) {
      const uint32_t stage = ptx::smem_u32(s.q[2 * half + ((c0 >> 5) & 1)]) + 32 * quad * 128;
      uint32_t o[32];
      ptx::tmem_ld32(tm_lane + H16Cols::O + 128 * half + c0, o);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * inv);
#pragma unroll
      for (int c = 0; c < 8; ++c)
        ptx::sts128(stage + lane * 128 + (uint32_t(c ^ (lane & 7)) << 4), o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 8; ++i) {  // rows 4 i + lane / 8
        const int r = 4 * i + (lane >> 3);
        const uint4 w = ptx::lds128(stage + r * 128 + (uint32_t((lane ^ r) & 7) << 4));
        if (32 * quad + r < live_rows)
          *reinterpret_cast<float4*>(orow + 4 * i * CKV + c0) = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
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
}

__global__ void __launch_bounds__(kH16Threads, 1) mla_decode_hm16_kernel(const DecodeParams P) {
  extern __shared__ uint8_t smem_raw[];
  H16Smem& s = *reinterpret_cast<H16Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(&s.full_a[i], 8), ptx::mbar_init(&s.full_b[i], 8);
      ptx::mbar_init(&s.free_a[i], 1), ptx::mbar_init(&s.free_b[i], 1);
    }
    ptx::mbar_init(&s.s_full, 1), ptx::mbar_init(&s.s_free, 8);
    ptx::mbar_init(&s.p_full, 8), ptx::mbar_init(&s.pv_done, 1);
    ptx::mbar_init(&s.q_full, 8);
    s.abort_flag = 0, s.progress = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 24) {
    ptx::tmem_alloc(&s.tmem_base, kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  ptx::tc_fence_after_sync();
  ptx::grid_dependency_wait();
  ptx::grid_launch_dependents();  // after the wait: the combine kernel reads a schedule kernel's output as soon as it starts
  // the query panels are free until the softmax warps write them
  if (P.inline_sched) publish_own_schedule<kH16Threads>(reinterpret_cast<int*>(s.q[0]), P, blockIdx.x >> 1);

  // register budgets, warp group by warp group; the pool is the launch allocation, 28 warps x 72
  constexpr int kLaunchRegs = 72, kSoftmaxRegs = 96, kConvertRegs = 64, kIssueRegs = 48;
  static_assert(8 * kSoftmaxRegs + 16 * kConvertRegs + 4 * kIssueRegs <= 28 * kLaunchRegs, "register budgets exceed the CTA's allocation");
  if (warp < 8) {
    ptx::reg_alloc<kSoftmaxRegs>();
    h16_run_role<kH16Softmax>(s, P);
  } else if (warp < 24) {
    ptx::reg_dealloc<kConvertRegs>();
    h16_run_role<kH16Convert>(s, P);
  } else {
    ptx::reg_dealloc<kIssueRegs>();
    if (warp == 24) h16_run_role<kH16Qk>(s, P);
    else if (warp == 25) h16_run_role<kH16Prefetch>(s, P);
    else if (warp == 26) h16_run_role<kH16Pv>(s, P);
    else h16_run_role<kH16Idle>(s, P);
  }

  ptx::tc_fence_before_sync();
  __syncthreads();
  if (warp == 24) ptx::tmem_dealloc(s.tmem_base, kTmemCols);
  if (threadIdx.x == 0 && s.abort_flag) atomicExch(P.header, int(kWaitTimeout));
}

}  // namespace mla
