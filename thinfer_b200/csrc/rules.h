// Index rules that kernels and launchers share and a CPU test compiles: no CUDA header in here.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TNF_HD __host__ __device__
#else
#define TNF_HD
#endif

namespace tnf {

// 128-row block of an operand's block scales that holds `row`; the last block there is for rows past the operand. A tile that
// hangs over the end of W copies that block once more: those columns are not stored, and the layout has nothing behind it.
TNF_HD inline uint32_t sf_row_block(uint32_t row, uint32_t rows) {
  const uint32_t last = (rows - 1u) >> 7, block = row >> 7;
  return block < last ? block : last;
}

// Width of the 1-CTA GEMM's 128-row tiles. 256 only when such tiles still fill the SMs and W has columns for more than half of
// one; 128-wide tiles also double-buffer the accumulator; with so few tiles that half the SMs would idle, 64-wide ones: a CTA's
// time is what it has to pull in (its A tile and its share of W) and what it writes out, and both shrink with the tile.
TNF_HD inline uint32_t tile_n_rule(uint32_t m, uint32_t n, uint32_t sms) {
  const uint64_t tm = (uint64_t(m) + 127u) / 128u;
  if (n > 128u && tm * ((uint64_t(n) + 255u) / 256u) >= sms) return 256u;
  return tm * ((uint64_t(n) + 127u) / 128u) * 2u <= sms ? 64u : 128u;
}

// Rows of the 1-CTA GEMM's tensor map over its packed activations ([m, k / 2] bytes). When many CTAs load through a map of less
// than 128 KB the loads are slow (K = 8192, N = 9216: 18.1 us for 31 rows, 11.3 for 32). Where there is `room` behind the operand
// the map reaches over it up to that size; the rows past m are loaded, multiplied and not stored. Measured (us, without / with):
// 16 x 9216 x 14336 SwiGLU 28.3 / 15.6, 1 x 16384 x 8192 22.0 / 13.3, 11 x 4096 x 4096 9.6 / 7.6, 11 x 2048 x 3072 7.0 / 6.8. A few
// CTAs only have the more rows to load, which cost more when they do not start on 128-byte lines: 38 x 304 x 2272 6.5 / 7.0,
// 11 x 2560 x 3168 7.5 / 8.2, 11 x 3584 x 3168 8.8 / 8.3.
constexpr uint64_t kSmallMapBytes = 128u << 10;
TNF_HD inline uint32_t map_rows_rule(uint32_t m, uint32_t n, uint32_t k, uint64_t room) {
  if (n < (k % 256u ? 3584u : 2048u)) return m;
  const uint64_t row = k / 2u, want = (kSmallMapBytes + row - 1u) / row, fit = room / row;
  const uint64_t rows = want < fit ? want : fit;
  return rows > m ? uint32_t(rows) : m;
}

// Rows of A that the 1-CTA GEMM's tiles load. The rows behind them in shared memory hold whatever they held: theirs are other rows of the
// accumulator, which are not stored. With 128 rows always, half of a K tile's bytes were A's whatever m was. Measured (us, 128 rows / these):
// 32 x 8640 x 8992 16.0 / 14.5, 64 x 9408 x 8992 with SwiGLU 17.1 / 15.8, 32 x 320 x 4768 with SwiGLU 8.6 / 7.85, 24 x 9408 x 12288 14.4 / 14.1.
TNF_HD inline uint32_t a_box_rule(uint32_t m) { return m <= 32u ? 32u : m <= 64u ? 64u : 128u; }
// The map claims no memory that is not there, not even to load nothing from it: one with further planes that were never loaded faulted.
// The map's rows for such boxes: where the map may reach past the operand at all it covers a whole box.
TNF_HD inline uint32_t a_map_rows(uint32_t m, uint32_t n, uint32_t k, uint64_t room) {
  const uint32_t rows = map_rows_rule(m, n, k, room), box = a_box_rule(m);
  if (n < (k % 256u ? 3584u : 2048u) || m > 64u || rows >= box) return rows;
  const uint64_t fit = room / (k / 2u);
  return fit >= box ? box : fit > rows ? uint32_t(fit) : rows;
}

// CTA pairs or single CTAs for an NVFP4 linear. A pair works on a 256 x 256 tile (or a half of it), the 1-CTA kernel on 128 x 128
// ones: while those fit one wave of CTAs they occupy more SMs, each for less time. Measured (us, quantiser included, pair against
// 1-CTA): 700 x 3072 x 3072 12.2 / 9.5, 300 x 6144 x 3072 12.2 / 9.2, 384 x 6144 x 12288 24.8 / 19.2; 130 shapes of all epilogues
// 1.42 times as fast in the geometric mean.
// In two waves the 1-CTA kernel reads its operands twice as often, and wins only while the pairs are not filled either, K is
// neither long (900 x 2560 x 8192 19.8 / 21.8) nor short (there a CTA's two epilogues are most of its time: 148 x 14608 x 288
// 8.1 / 9.2, 2331 x 1248 x 608 9.9 / 10.4), the epilogue reads no residual (186 x 10592 x 1024 10.7 / 11.6) and there are more than
// two rows of tiles (199 x 11120 x 1024 8.1 / 8.5). Then: 893 x 3472 x 1024 9.4 / 8.4, 447 x 9408 x 2048 with GELU 12.2 / 10.7.
// Outputs that are also stored to peers go out in the pair kernel's 128-byte row segments, which NVLink packs well, whenever there
// are pair tiles for most of the chip.
TNF_HD inline bool pair_rule(uint32_t m, uint32_t n, uint32_t k, bool gated, bool peers, uint32_t sms) {
  if (m <= 128u) return false;
  const uint64_t tiles1 = ((uint64_t(m) + 127u) / 128u) * ((uint64_t(n) + 127u) / 128u);
  const uint64_t tiles2 = ((uint64_t(m) + 255u) / 256u) * ((uint64_t(n) + 255u) / 256u);
  if (peers) return tiles2 >= 32u;
  if (tiles1 <= sms) return false;
  return !(tiles2 <= sms / 2u && k > 768u && k <= 2048u && m > 256u && !gated);
}

// Width of the 1-CTA kernel's tiles for the dense arm, 0 for the pair kernel: the narrowest that leaves one wave. A CTA's time is its K loop,
// which the issue of small MMAs bounds (55-60 cycles each up to 64 columns, 80-90 with 128), and the weight of few rows comes in faster the more
// CTAs have loads in flight. In two waves the pair kernel is the better one (300 x 9216 x 3072 20.1 / 22.8, 512 x 9216 x 14336 89 / 114). Measured
// (us, pair kernel / these): 16 x 3072 x 3072 12.2 / 8.2, 64 x 4736 x 14336 69.9 / 27.8, 128 x 9216 x 3072 14.5 / 10.4, 512 x 4736 x 3072 18.5 / 13.6,
// 1 x 256 x 512 4.8 / 3.2; 150 shapes 1.8 times as fast in the geometric mean, the least 1.06 (292 x 4096 x 2976 15.2 / 14.3).
TNF_HD inline uint32_t dense_tile_rule(uint32_t m, uint32_t n, bool quantised, uint32_t sms) {
  const uint64_t tm = (uint64_t(m) + 127u) / 128u;
  for (uint32_t bn = quantised ? 64u : 32u; bn <= 128u; bn *= 2u)
    if (tm * ((uint64_t(n) + bn - 1u) / bn) <= sms) return bn;
  return 0u;
}

// With up to 16 rows clusters of CTAs also share K, in stages of 256 elements with 32 columns, else of 128. Cycles: what 64 elements of K take a
// CTA, or the weight from HBM where that is more, and for the join a start and every further CTA's sums. Only where that leaves four
// fifths, and in clusters of 2, 4 or 8: of 3, 5 and 6 too few fit beside the launch before (1600 columns in clusters of five, K = 3072: 7.6 us alone,
// 9.2). Measured (us, alone / clusters): 16 x 256 x 14336 25.2 / 6.8, 1 x 1024 x 3072 7.6 / 5.7, 16 x 1024 x 9216 17.3 / 7.9, 8 x 3072 x 6144 13.6 / 10.9,
// 16 x 2048 x 14336 25.7 / 12.7; 210 shapes 1.29 times as fast in the geometric mean, the least 0.98; not taken: 16 x 2048 x 1024 4.3 / 5.2,
// 16 x 9216 x 9216 29.5 / 30.8.
struct DenseTiles {
  uint32_t bn, ctas, share;  // bn 0: the pair kernel; ctas 1: no clusters; stages of each CTA
};
inline DenseTiles dense_tiles_rule(uint32_t m, uint32_t n, uint32_t k, bool quantised, uint32_t sms, const int* clusters) {
  DenseTiles t{dense_tile_rule(m, n, quantised, sms), 1u, 0u};
  if (m > 16u || !t.bn) return t;
  const uint64_t boxes = (k + 63u) / 64u, hbm = uint64_t(n) * k / 1750u;
  auto loop = [&](uint32_t bn, uint64_t b) {
    const uint64_t c = b * (bn == 32u ? 220u : bn == 64u ? 270u : 330u);
    return c > hbm ? c : hbm;
  };
  uint64_t best = loop(t.bn, boxes) * 4u / 5u;
  for (uint32_t bn = quantised ? 64u : 32u; bn <= 128u; bn *= 2u)
    for (uint32_t c = 2; c <= 8u; c *= 2u) {
      const uint32_t per = bn == 32u ? 4u : 2u, stages = (uint32_t(boxes) + per - 1u) / per, share = (stages + c - 1u) / c, ctas = (stages + share - 1u) / share;
      if (clusters[c] < 0 || (n + bn - 1u) / bn > uint32_t(clusters[c]) || ctas != c) continue;
      const uint64_t cost = loop(bn, share * per) + 2600u + (c - 1u) * (bn / 32u) * 220u;
      if (cost >= best) continue;
      best = cost;
      t = DenseTiles{bn, c, share};
    }
  return t;
}

// CTAs of a cluster that share the K tiles (256 elements) of 128 output columns of a linear of up to 16 rows, 1 for none, and the K tiles
// of each. `clusters[n]`: clusters of n CTAs that are on the device at once; all have to be. `one_launch`: the call would otherwise take
// the skinny kernel without clusters, else quantiser and GEMM. The costs are fitted (10 ns) to 400 shapes of 1 to 16 rows, which the
// split makes 1.27 times as fast in the geometric mean, the best choice for each 1.27: a start, and per K tile of a CTA its weight and the
// quantisation of its activations (with 256 threads for up to four rows, 512 for more). Measured (us, without / with clusters): 1 x 3072 x 3072 5.6 /
// 4.2, 16 x 3072 x 3072 6.8 / 6.0, 1 x 256 x 14336 28.6 / 4.7, 4 x 9216 x 9216 19.8 / 9.8, 16 x 9216 x 14336 28.4 / 17.7; not taken: 4 x 6144 x 1024
// 3.9 / 4.1, 1 x 4736 x 512 3.2 / 3.5, 16 x 6144 x 2048 6.3 / 6.5, 16 x 256 x 512 4.98 / 4.8.
// SwiGLU, which would otherwise always take two launches: 150 shapes 1.44 times as fast, none slower (1 x 3072 x 3072 6.8 / 4.0, 8 x 9216 x 3072 8.2 /
// 6.5, 1 x 9216 x 14336 28.8 / 10.2, 16 x 9216 x 14336 28.8 / 17.7).
struct SkinnySplit {
  uint32_t ctas, share;
};
inline uint32_t skinny_split_threads(uint32_t m) { return m <= 4u ? 256u : 512u; }
inline SkinnySplit skinny_split_rule(uint32_t m, uint32_t n, uint32_t k, bool one_launch, const int* clusters) {
  const uint32_t tiles = (n + 127u) / 128u, nkt = (k + 255u) / 256u;
  const uint64_t per_tile = 84u + 12u * m;  // quarter units: 21 + 3 m
  uint64_t best = 4u * (one_launch ? 290u : 440u) + nkt * (one_launch ? per_tile : tiles >= 32u ? 136u : 72u);
  SkinnySplit s{1u, 0u};
  for (uint32_t c = 2; c <= 8u; ++c) {
    if (clusters[c] < 0 || tiles > uint32_t(clusters[c]) || nkt < (m <= 4u ? 6u : 4u) || nkt < c || (c == 2u && nkt < (m <= 4u ? 8u : 12u))) continue;
    const uint32_t share = (nkt + c - 1u) / c;
    const uint64_t cost = m <= 4u ? 4u * 340u + share * per_tile : 4u * (350u + 4u * m) + share * uint64_t(84u + 7u * m);
    if (cost >= best) continue;
    best = cost;
    s = SkinnySplit{(nkt + share - 1u) / share, share};
  }
  return s;
}

// Tiles that the pair kernel takes whole; each later one runs as two halves of 128 columns. The last wave's are split when every half
// then finds a pair of its own (and none is empty). An only wave would be split as well, but calls of so few tiles
// take the 1-CTA kernel. Not with stores to other GPUs, whose row segments a half would shorten (not measured).
TNF_HD inline uint32_t pair_whole_tiles(uint32_t tiles, uint32_t n, uint32_t pairs, bool remote) {
  const uint32_t tail = tiles % pairs;
  const bool split = tail > 0u && 2u * tail <= pairs && n % 256u == 0u && !(remote && tiles <= pairs);
  return split ? tiles - tail : tiles;
}

// Whether a plain or an NVFP4 output (local, no residual) takes its own epilogue, which shortens a tile that the epilogue bounds, or the
// general one. With a long K the tile is bound by its main loop, and the general one, whose stores are spread over more of it,
// disturbs the loop less. Measured (us, general / own): plain 4257 x 1120 x 768 10.9 / 10.2, 3352 x 2992 x 1280 15.8 / 15.3, 4137 x 7280 x 2048
// 35.5 / 36.3; GELU 5394 x 10640 x 1280 54.8 / 48.2, 5434 x 4144 x 2048 32.5 / 30.2, 6013 x 4416 x 4096 59.1 / 59.7; NVFP4 4601 x 7168 x 1792
// 35.3 / 31.5, 3716 x 12096 x 3072 60.6 / 61.6; GELU + NVFP4 3228 x 18176 x 3584 91.4 / 89.3, 8456 x 11968 x 6144 248.7 / 248.2. In less than two
// waves the last epilogue is not hidden at all: plain 1612 x 1520 x 2560 12.1 / 11.7, GELU 4129 x 944 x 9216 37.0 / 36.4. The dense arm takes
// four times as long for a K.
TNF_HD inline bool pair_epilogue_rule(uint32_t k, bool dense, bool gelu, bool quantised, uint32_t tiles, uint32_t pairs) {
  if (tiles < 2u * pairs || (quantised && gelu)) return true;
  const uint64_t k4 = dense ? uint64_t(k) * 4u : k;
  return k4 < (quantised ? 3072u : gelu ? 3584u : 2048u);
}

// Work items of the attention kernel. A (head, batch) pair has ceil(s_q / 128) blocks of 128 query rows; two of them make a tile.
// An item is a tile (rows mode: one softmax group per block, all keys each) or one block (keys mode: the groups share the keys),
// which takes about half as long. Items [0, full_items) are tiles, the others the blocks of the tiles that are left and then, where
// the number of blocks is odd, the last block of every pair.
// The slowest CTA gets the number of half waves that the blocks make, no more: the tiles left over after whole waves are taken as
// blocks when all that is left over fits one half wave. Otherwise they stay tiles (which read K and V once for 256 rows) and the
// odd blocks go to the CTAs that have no tile in that wave, two each, then to all in turn. Counting an odd block as a tile instead
// costs up to a half wave: 1111 x 1500 keys x 16 heads 25.4 against 16.1 us, 2 x 300 x 4000 x 24 57.3 against 42.1.
struct SdpaPlan {
  uint32_t pair_tiles;  // whole tiles of a (head, batch) pair
  uint32_t full_items, odd_first, items;  // tiles; blocks of tiles; from odd_first on the pairs' odd blocks
  uint32_t ctas, skip;  // CTAs; the first `skip` of them have a tile more than the others
};
struct SdpaSlot {
  uint32_t pair, q_first, keys_mode;  // (head, batch) pair, first query row, one block with shared keys
};
// False when there are too many items to number.
inline bool sdpa_plan(uint32_t s_q, uint64_t pairs, uint32_t sms, SdpaPlan* p) {
  const uint64_t blocks = (uint64_t(s_q) + 127u) / 128u, tiles = pairs * (blocks / 2u), odd = pairs * (blocks & 1u);
  const uint64_t tail = tiles % sms, full = 2u * tail + odd <= sms ? tiles - tail : tiles, items = full + 2u * (tiles - full) + odd;
  if (items > 0x7FFFFFFFull) return false;
  p->pair_tiles = uint32_t(blocks / 2u);
  p->full_items = uint32_t(full);
  p->odd_first = uint32_t(items - odd);
  p->items = uint32_t(items);
  p->ctas = items < sms ? uint32_t(items) : sms;
  p->skip = p->full_items % p->ctas;
  return true;
}
// CTAs of a cluster that share the keys of one block, 1 for none; `clusters[n]`: clusters of n CTAs that are on the device at once. Few
// blocks leave SMs idle: all blocks have to be on the chip at once, and of the sizes that allow it the one with the fewest key
// tiles a CTA wins, the two groups' tiles counted in pairs. Joining the outputs costs about what four tiles take (2.6 us). Measured
// (us, blocks x key tiles, one CTA / so many): 1 x 8 11.5 / 9.3 (4), 16 x 8 12.0 / 10.0 (4), 64 x 8 12.7 / 13.0 (2, not taken), 8 x 32 30.7 / 13.4 (8),
// 24 x 32 31.3 / 16.6 (5), 48 x 16 19.0 / 16.7 (2), 48 x 128 108 / 74 (2). More CTAs than fit at once never won.
inline uint32_t sdpa_split(uint64_t blocks, uint32_t s_k, const int* clusters) {
  const uint32_t tiles = (s_k + 127u) / 128u;
  uint32_t best = 1u, cost = tiles;
  for (uint32_t n = 2; n <= 8u && tiles >= 2u * n; ++n) {
    const uint32_t share = (tiles + n - 1u) / n, c = (share + 1u) / 2u * 2u + 4u;
    if (clusters[n] < 0 || blocks > uint64_t(clusters[n]) || c >= cost) continue;
    best = n;
    cost = c;
  }
  return best;
}
// Its plan: every block an item, a cluster each.
inline void sdpa_split_plan(uint32_t s_q, uint64_t pairs, SdpaPlan* p) {
  const uint64_t blocks = (uint64_t(s_q) + 127u) / 128u, items = pairs * blocks;
  *p = SdpaPlan{uint32_t(blocks / 2u), 0u, uint32_t(items - pairs * (blocks & 1u)), uint32_t(items), uint32_t(items), 0u};
}
// The items of a CTA: sdpa_first, then sdpa_next until it is not below `items`.
TNF_HD inline uint32_t sdpa_first_block(const SdpaPlan& p, uint32_t cta) {
  return p.full_items + (cta >= p.skip ? cta - p.skip : 2u * (p.ctas - p.skip) + cta);
}
TNF_HD inline uint32_t sdpa_first(const SdpaPlan& p, uint32_t cta) { return cta < p.full_items ? cta : sdpa_first_block(p, cta); }
TNF_HD inline uint32_t sdpa_next(const SdpaPlan& p, uint32_t cta, uint32_t it) {
  if (it < p.full_items) return it + p.ctas < p.full_items ? it + p.ctas : sdpa_first_block(p, cta);
  const uint32_t block = it - p.full_items, idle = p.ctas - p.skip;
  if (block < idle) return it + idle;
  return block < 2u * idle ? p.full_items + 2u * idle + cta : it + p.ctas;
}
TNF_HD inline SdpaSlot sdpa_slot(const SdpaPlan& p, uint32_t it) {
  if (it >= p.odd_first) return SdpaSlot{it - p.odd_first, p.pair_tiles * 256u, 1u};
  const uint32_t keys_mode = it >= p.full_items ? 1u : 0u, block = keys_mode ? it - p.full_items : 0u;
  const uint32_t tile = keys_mode ? p.full_items + (block >> 1) : it, pair = tile / p.pair_tiles;
  return SdpaSlot{pair, (tile - pair * p.pair_tiles) * 256u + (block & 1u) * 128u, keys_mode};
}

}  // namespace tnf
