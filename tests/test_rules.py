"""The index rules that kernels and launchers share (csrc/rules.h), compiled for the CPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include "rules.h"
extern "C" {
uint32_t row_block(uint32_t row, uint32_t rows) { return tnf::sf_row_block(row, rows); }
uint32_t tile_n(uint32_t m, uint32_t n, uint32_t sms) { return tnf::tile_n_rule(m, n, sms); }
int pair(uint32_t m, uint32_t n, uint32_t k, int gated, int peers, uint32_t sms) { return tnf::pair_rule(m, n, k, gated != 0, peers != 0, sms); }
int own_epilogue(uint32_t k, int dense, int gelu, int q, uint32_t tiles, uint32_t pairs) { return tnf::pair_epilogue_rule(k, dense != 0, gelu != 0, q != 0, tiles, pairs); }
uint32_t map_rows(uint32_t m, uint32_t n, uint32_t k, uint64_t room) { return tnf::map_rows_rule(m, n, k, room); }
uint32_t a_box(uint32_t m) { return tnf::a_box_rule(m); }
uint32_t a_rows(uint32_t m, uint32_t n, uint32_t k, uint64_t room) { return tnf::a_map_rows(m, n, k, room); }
uint32_t whole_tiles(uint32_t tiles, uint32_t n, uint32_t pairs, int remote) { return tnf::pair_whole_tiles(tiles, n, pairs, remote != 0); }
// items of every CTA in its order, as {cta, pair, q_first, keys_mode}; the number of CTAs, or -1 when there are too many items
int64_t sdpa_items(uint32_t s_q, uint64_t pairs, uint32_t sms, uint32_t* out, uint64_t* n, uint64_t room) {
  tnf::SdpaPlan p{};
  *n = 0;
  if (!tnf::sdpa_plan(s_q, pairs, sms, &p)) return -1;
  for (uint32_t c = 0; c < p.ctas; ++c)
    for (uint32_t it = tnf::sdpa_first(p, c); it < p.items && *n < room; it = tnf::sdpa_next(p, c, it)) {
      const tnf::SdpaSlot s = tnf::sdpa_slot(p, it);
      uint32_t* o = out + 4 * (*n)++;
      o[0] = c; o[1] = s.pair; o[2] = s.q_first; o[3] = s.keys_mode;
    }
  return p.ctas;
}
void skinny(uint32_t m, uint32_t n, uint32_t k, int one, const int* clusters, uint32_t* out) {
  const tnf::SkinnySplit s = tnf::skinny_split_rule(m, n, k, one != 0, clusters);
  out[0] = s.ctas; out[1] = s.share;
}
uint32_t dense_tile(uint32_t m, uint32_t n, int q, uint32_t sms) { return tnf::dense_tile_rule(m, n, q != 0, sms); }
void dense_tiles(uint32_t m, uint32_t n, uint32_t k, int q, uint32_t sms, const int* clusters, uint32_t* out) {
  const tnf::DenseTiles t = tnf::dense_tiles_rule(m, n, k, q != 0, sms, clusters);
  out[0] = t.bn; out[1] = t.ctas; out[2] = t.share;
}
uint32_t split(uint64_t blocks, uint32_t s_k, const int* clusters) { return tnf::sdpa_split(blocks, s_k, clusters); }
void split_items(uint32_t s_q, uint64_t pairs, uint32_t* out) {  // {pair, q_first, keys_mode} of every item
  tnf::SdpaPlan p{};
  tnf::sdpa_split_plan(s_q, pairs, &p);
  for (uint32_t it = 0; it < p.items; ++it) {
    const tnf::SdpaSlot s = tnf::sdpa_slot(p, it);
    out[3 * it] = s.pair; out[3 * it + 1] = s.q_first; out[3 * it + 2] = s.keys_mode;
  }
}
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "librules.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(ROOT, "thinfer_b200", "csrc"), "-o", str(so),
                    str(d / "shim.cpp")], check=True)
    return C.CDLL(str(so))


def test_no_tile_copies_scales_past_the_weight(rules):
    """The scale layout of W ends with the 128-row block of its last row: whatever the tile's width, every block that it copies
    is one of those, and the right one wherever W has rows."""
    past = 0
    for m in (1, 128, 129, 256, 385, 512, 1000, 9345, 18817, 18944, 40000):
        for n in (8, 64, 128, 136, 256, 264, 384, 9216, 9224, 9344, 9352, 18688, 18696, 18816, 37632, 37640, 37760, 37888, 40000):
            width = rules.tile_n(m, n, 148)
            blocks = (n + 127) // 128
            assert width in (64, 128, 256)
            assert width <= 128 or n > 128  # half of a 256-wide tile would be padding in every CTA
            for n0 in range(0, n, width):
                for j in range(max(1, width // 128)):
                    row = n0 + 128 * j
                    block = rules.row_block(row, n)
                    assert block < blocks
                    if row < n:
                        assert block == row // 128
                    past += row // 128 >= blocks
    assert past > 0  # there are shapes here whose last tile hangs over by a whole block


def test_map_over_few_rows_stays_inside_the_buffer(rules):
    for k in (32, 96, 256, 3072, 8192, 8992, 14336, 65536, 262144 + 32, 1 << 20):
        for m in (1, 16, 17, 31, 32, 100, 128, 5000):
            need = m * k // 2
            for room in (0, need, need + k // 2, (128 << 10) + k // 2, 16 << 20, 1 << 40):
                rows = rules.map_rows(m, 4096, k, C.c_uint64(room))
                assert rules.map_rows(m, 1024, k, C.c_uint64(room)) == m
                assert rows >= m
                assert rows == m or rows * k // 2 <= room
                assert rows == m or (rows - 1) * k // 2 < 128 << 10  # no taller than it has to be
                if room >= (128 << 10) + k // 2:
                    assert rows * k // 2 >= 128 << 10


def test_boxes_over_few_rows(rules):
    """A box holds every row of its tile; the map covers the box where the buffer has room and never more than the buffer."""
    for k in (32, 96, 3072, 8992, 14336, 1 << 20):
        for m in (1, 16, 17, 32, 33, 64, 65, 128, 129, 5000):
            box = rules.a_box(m)
            assert box in (32, 64, 128) and box >= min(m, 128)
            for n in (256, 4096):
                for room in (0, m * k // 2, box * k // 2, (128 << 10) + k // 2, 1 << 40):
                    rows = rules.a_rows(m, n, k, C.c_uint64(room))
                    assert rows >= m and (rows == m or rows * k // 2 <= room)
                    if n == 4096 and m <= 64 and room >= box * k // 2:
                        assert rows >= box


def test_epilogue_of_the_pair_kernel(rules):
    own = lambda k, dense=0, gelu=0, q=0, tiles=148, pairs=74: bool(rules.own_epilogue(k, dense, gelu, q, tiles, pairs))
    assert own(2047) and not own(2048) and own(511, dense=1) and not own(512, dense=1)
    assert own(3583, gelu=1) and not own(3584, gelu=1) and own(895, dense=1, gelu=1) and not own(896, dense=1, gelu=1)
    assert own(3071, q=1) and not own(3072, q=1) and own(1 << 20, gelu=1, q=1)
    assert own(1 << 30, dense=1, tiles=147)  # less than two waves: the last epilogue shows whatever K is


def test_halves_of_pair_tiles(rules):
    """No more items than pairs in the last wave, no empty half, and no halves in the only wave of an output that goes to other GPUs."""
    for pairs in (74, 3):
        for tiles in range(1, 4 * pairs + 1):
            for n in (256, 3072, 3080):
                for remote in (0, 1):
                    whole = rules.whole_tiles(tiles, n, pairs, remote)
                    halves = 2 * (tiles - whole)
                    assert whole == tiles or (n % 256 == 0 and whole % pairs == 0 and 0 < halves <= pairs)
                    if tiles <= pairs:
                        assert (whole == tiles) == (bool(remote) or n % 256 != 0 or 2 * tiles > pairs)


def test_outputs_to_peers_take_the_pair_kernel(rules):
    """The pair kernel stores to peers in 128-byte row segments: such calls take it from 32 of its tiles on, whatever is the better
    kernel for a local output."""
    differ = 0
    for m in (1, 128, 129, 256, 300, 700, 1024, 4352):
        for n in (256, 3072, 6144, 9472, 18432):
            for k in (256, 2048, 12288):
                tiles = -(-m // 256) * -(-n // 256)
                assert rules.pair(m, n, k, 0, 1, 148) == (m > 128 and tiles >= 32), (m, n, k)
                differ += rules.pair(m, n, k, 0, 1, 148) != rules.pair(m, n, k, 0, 0, 148)
    assert differ > 0


@pytest.mark.parametrize("m,n,k,gated,pair", [
    (700, 3072, 12288, 0, 0), (700, 3072, 12288, 1, 0), (130, 9472, 64, 0, 0),  # one wave of 128 x 128 tiles: single CTAs
    (893, 3472, 1024, 0, 0), (447, 9408, 2048, 0, 0), (2111, 1520, 1536, 0, 0),  # two waves, K neither short nor long
    (893, 3472, 1024, 1, 1),                                                     # ... with a gated residual
    (148, 14608, 288, 0, 1), (2331, 1248, 608, 0, 1), (900, 2560, 8192, 0, 1),   # K short or long
    (199, 11120, 1024, 0, 1), (4352, 3072, 1024, 0, 1),                          # two rows of tiles; the pairs are filled
])
def test_kernel_of_measured_shapes(rules, m, n, k, gated, pair):
    assert rules.pair(m, n, k, gated, 0, 148) == pair


@pytest.mark.parametrize("sms", [148, 7])
@pytest.mark.parametrize("s_q", [1, 17, 128, 129, 256, 257, 300, 384, 385, 512, 640, 1111, 2000, 4352])
def test_attention_items(rules, s_q, sms):
    """Every block of 128 query rows of every (head, batch) pair is in exactly one item, no item is empty, every CTA has one, and
    the slowest CTA takes the least number of half waves that the blocks allow."""
    rules.sdpa_items.restype = C.c_int64
    blocks = -(-s_q // 128)
    for pairs in (1, 2, 3, 8, 12, 16, 24, 37, 48, 80, 147, 148, 149, 300, 500):
        room = pairs * blocks
        out, n = np.zeros((room + 1, 4), np.uint32), C.c_uint64()
        ctas = rules.sdpa_items(C.c_uint32(s_q), C.c_uint64(pairs), C.c_uint32(sms), out.ctypes.data_as(C.c_void_p), C.byref(n), C.c_uint64(room + 1))
        assert 0 < ctas <= sms and n.value <= room
        items = out[: n.value].astype(np.int64)
        seen = np.zeros((pairs, blocks), np.int64)
        for half in (0, 1):  # a tile is two blocks
            rows = items[(items[:, 3] == 0) | (half == 0)]
            assert (rows[:, 2] % 128 == 0).all()
            np.add.at(seen, (rows[:, 1], rows[:, 2] // 128 + half), 1)  # raises on a block that does not exist
        assert (seen == 1).all(), (pairs, s_q)
        halves = np.bincount(items[:, 0], weights=np.where(items[:, 3] == 0, 2, 1), minlength=ctas)
        assert (halves > 0).all()
        best = -(-pairs * blocks // sms)
        assert halves.max() == best, (pairs, halves.max(), best)


def test_attention_items_are_numbered_in_31_bits(rules):
    rules.sdpa_items.restype = C.c_int64
    n = C.c_uint64()
    assert rules.sdpa_items(C.c_uint32((1 << 31) - 1), C.c_uint64(256), C.c_uint32(148), None, C.byref(n), C.c_uint64(0)) == -1
    assert rules.sdpa_items(C.c_uint32(1 << 20), C.c_uint64(65535), C.c_uint32(148), None, C.byref(n), C.c_uint64(0)) == 148


def test_shares_of_the_keys(rules):
    """Clusters only where all of them fit the chip at once, with two key tiles at least for every CTA, and a cheaper share."""
    fit = (C.c_int * 9)(0, 0, 74, 45, 36, 27, 20, 14, 14)
    split = lambda blocks, s_k: rules.split(C.c_uint64(blocks), C.c_uint32(s_k), fit)
    for blocks in (1, 7, 14, 15, 20, 21, 36, 37, 45, 46, 74, 75, 148, 1 << 40):
        for tiles in range(1, 140):
            n = split(blocks, tiles * 128 - 5)
            assert n == split(blocks, tiles * 128) and 1 <= n <= 8
            if n > 1:
                assert blocks <= fit[n] and tiles >= 2 * n and -(-tiles // n) + 4 <= tiles
            if blocks > 74 or tiles < 8:
                assert n == 1
    assert split(1, 1024) == 4 and split(64, 1024) == 1 and split(14, 4096) == 8 and split(48, 2048) == 2 and split(45, 4096) == 3
    none = (C.c_int * 9)()
    assert rules.split(C.c_uint64(1), C.c_uint32(1 << 20), none) == 1


def test_every_block_has_a_cluster(rules):
    for s_q in (1, 128, 129, 256, 300, 520, 1111):
        for pairs in (1, 3, 10):
            blocks = (s_q + 127) // 128
            out = np.zeros((pairs * blocks, 3), np.uint32)
            rules.split_items(C.c_uint32(s_q), C.c_uint64(pairs), out.ctypes.data_as(C.c_void_p))
            assert sorted((int(p), int(q)) for p, q, _ in out) == [(p, 128 * b) for p in range(pairs) for b in range(blocks)]
            assert (out[:, 2] == 1).all()


def test_shares_of_k(rules):
    """Clusters for a few rows: all of them on the chip at once, every CTA with a K tile, all K tiles covered, and no more CTAs than that."""
    fit = (C.c_int * 9)(0, 0, 74, 45, 36, 27, 20, 14, 14)
    out = (C.c_uint32 * 2)()

    def split(m, n, k, one, counts=fit):
        rules.skinny(C.c_uint32(m), C.c_uint32(n), C.c_uint32(k), int(one), counts, out)
        return out[0], out[1]
    seen = set()
    for m in range(1, 17):
        for n in (8, 128, 136, 1024, 3072, 4736, 4744, 6144, 9472, 9480, 18432, 1 << 20):
            for k in (32, 256, 288, 1024, 1312, 2048, 3072, 4128, 9216, 14336, 1 << 20):
                for one in (False, True):
                    ctas, share = split(m, n, k, one)
                    seen.add(ctas)
                    nkt, tiles = -(-k // 256), -(-n // 128)
                    if ctas > 1:
                        assert tiles <= fit[ctas] and ctas * share >= nkt > (ctas - 1) * share
                    assert split(m, n, k, one, (C.c_int * 9)())[0] == 1
    assert seen >= {1, 2, 3, 4, 5, 6, 8}
    assert split(1, 3072, 3072, True) == (4, 3) and split(4, 9216, 9216, False) == (2, 18)  # measured choices ...
    assert split(4, 6144, 1024, True)[0] == 1 and split(1, 4736, 512, True)[0] == 1         # ... and what lost


def test_dense_tiles(rules):
    """The 1-CTA kernel takes the dense arm in one wave of its tiles, with 64 columns at least where they are quantised; clusters only for up
    to 16 rows, all of them on the chip at once, every CTA with a stage of K, all stages covered."""
    fit, none, out = (C.c_int * 9)(0, 0, 74, 45, 36, 27, 20, 14, 14), (C.c_int * 9)(), (C.c_uint32 * 3)()
    seen = set()
    for sms in (148, 7):
        for m in (1, 5, 16, 17, 64, 128, 129, 512, 1200, 6400, 9600, 1 << 20):
            for n in (8, 64, 256, 320, 1040, 2048, 3072, 4736, 9216, 18944, 18952, 1 << 20):
                for q in (0, 1):
                    bn, wave = rules.dense_tile(m, n, q, sms), lambda width: -(-m // 128) * -(-n // width) <= sms
                    assert bn in (0, 32, 64, 128) and not (q and bn == 32)
                    assert wave(bn) if bn else not wave(128)
                    assert bn in (0, 64 if q else 32) or not wave(bn // 2)  # the narrowest
                    for k in (32, 96, 512, 1120, 3072, 9216, 14336, 1 << 20):
                        for counts in (fit, none):
                            rules.dense_tiles(C.c_uint32(m), C.c_uint32(n), C.c_uint32(k), q, C.c_uint32(sms), counts, out)
                            width, ctas, share = out
                            if ctas == 1:
                                assert width == bn
                                continue
                            assert m <= 16 and bn and ctas in (2, 4, 8) and width in (32, 64, 128) and not (q and width == 32)
                            stages = -(-k // (256 if width == 32 else 128))
                            assert (ctas - 1) * share < stages <= ctas * share
                            assert -(-n // width) <= counts[ctas]
                            seen.add((width, ctas))
    assert {c for _, c in seen} == {2, 4, 8} and {w for w, _ in seen} == {32, 64, 128}
