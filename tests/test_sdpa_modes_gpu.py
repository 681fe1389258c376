"""Attention with more blocks of 128 query rows than SMs: items of 256 rows (one softmax group per 128) and of 128 rows whose groups
share the keys, several a CTA, in the mixtures that sdpa_plan (csrc/rules.h; its own test is test_rules.py) makes. Against the restated reference, same tolerance and reason as
test_sdpa_gpu.py (bf16 probabilities in the second product, bf16 inputs and outputs)."""
import numpy as np
import pytest

import oracle as O
from conftest import dev_scales_to_canonical, rel_fro
from test_sdpa_gpu import TOL, _inputs, _run

pytestmark = pytest.mark.gpu
SCALE = float(1.0 / np.sqrt(128.0))


@pytest.mark.parametrize("b,s_q,s_k,h_q,h_kv,spread", [
    (1, 300, 200, 80, 80, 1.0),    # 80 tiles, and 80 blocks of 44 rows on the other 68 CTAs: two on twelve of them
    (2, 520, 330, 30, 10, 1.0),    # 120 tiles, 60 blocks of 8 rows: two on each of the other 28 CTAs, four after tiles; grouped heads; two batches
    (1, 129, 700, 100, 100, 1.0),  # tiles only; the second group has one row
    (1, 100, 17, 100, 50, 1.0),    # one ragged key tile: the second group has none
    (1, 256, 1024, 76, 76, 6.0),   # peaked rows: the running output of both groups is rescaled from tile to tile
    (1, 100, 17, 310, 310, 1.0),   # blocks only, three a CTA, the second group without a key tile
    (1, 100, 130, 150, 150, 6.0),  # blocks only, two a CTA on two of them; two keys more than one tile
    (1, 70, 1300, 150, 50, 1.0),   # ... with eleven key tiles: both rings go round several times in the second item, too
    (1, 1111, 150, 60, 20, 1.0),   # a wave of tiles, 92 more, and 60 blocks of 87 rows on the other 56 CTAs
    (1, 1111, 400, 37, 37, 1.0),   # a whole wave of tiles, then 37 blocks
    (1, 300, 64, 140, 70, 1.0),    # 140 tiles and as many blocks of 44 rows: 16 on the idle CTAs, the others after tiles
    (1, 300, 150, 300, 300, 1.0),  # two waves of tiles and four; 300 blocks: two on 144 CTAs, 12 more on the first
])
def test_rows_mode_matches_reference_recurrence(backend, b, s_q, s_k, h_q, h_kv, spread):
    q, k, v = _inputs(b, s_q, s_k, h_q, h_kv, 31 * s_q + s_k, spread)
    got = O.bf16_to_f32(_run(backend, q, k, v, SCALE))
    want = O.bf16_to_f32(O.ref_sdpa(q, k, v, SCALE))
    assert not np.isnan(got).any()
    for bi in range(b):  # per head: an error in one CTA's tile must not hide in the norm over all of them
        for h in range(h_q):
            assert rel_fro(got[bi, :, h], want[bi, :, h]) <= 1.25 * TOL, (bi, h)
    assert rel_fro(got, want) <= TOL


@pytest.mark.parametrize("s_q,heads", [(130, 1), (256, 80)])  # keys mode, rows mode
@pytest.mark.parametrize("jumps", [
    {127: 400.0},                             # the first tile's last key decides the reference maximum
    {128: 12.0, 256 + 95: 24.0},              # just past the limit, in the keys whose sum is checked
    {128 + 96: 12.0, 256 + 127: 24.0},        # ... in the last 32 keys, whose maximum is checked
    {130: 300.0, 300: 600.0, 511: 900.0},     # probabilities would overflow f32 against the older maximum
    {5: 900.0},                               # everything after the first tile underflows to zero
])
def test_scores_that_jump(backend, s_q, heads, jumps):
    """Score of key j (exp2 domain) = jumps[j], small noise elsewhere, the same for every row."""
    s_k, d = 520, 128
    rng = np.random.default_rng(7)
    k = np.zeros((1, s_k, heads, d), np.float32)
    k[..., 0] = rng.uniform(-1, 1, (1, s_k, heads))
    for j, x in jumps.items():
        k[:, j, :, 0] = x
    q = np.zeros((1, s_q, heads, d), np.float32)
    q[..., 0] = np.log(2.0) / SCALE
    v = rng.standard_normal((1, s_k, heads, d)).astype(np.float32)
    q, k, v = (O.f32_to_bf16(t) for t in (q, k, v))
    got, want = O.bf16_to_f32(_run(backend, q, k, v, SCALE)), O.bf16_to_f32(O.ref_sdpa(q, k, v, SCALE))
    assert not np.isnan(got).any() and rel_fro(got, want) <= TOL


def test_rows_mode_fused_output_quantisation(backend):
    be, (s, heads) = backend, (300, 80)
    cols = heads * 128
    q, k, v = _inputs(1, s, s, heads, heads, 512)
    plain = _run(be, q, k, v, SCALE).reshape(s, cols)
    g = O.global_scale(O.amax_bf16(plain))
    qb, kb, vb = be.upload(q), be.upload(k), be.upload(v)
    want_c, want_s = O.quantize_act(plain, g)
    want_dev = O.scales_to_device_layout(want_s)
    codes, scales = be.allocate(s * cols // 2), be.upload(np.full(want_dev.size, 0x7F, np.uint8))
    be.scope().sdpa(qb, kb, vb, None, 1, s, s, heads, heads, SCALE, out_nvfp4=(codes, scales, g))
    be.submit(30000)
    assert np.array_equal(be.read_buffer(codes).reshape(s, cols // 2), want_c)
    dev = be.read_buffer(scales)
    assert np.array_equal(dev_scales_to_canonical(dev, s, cols), want_s) and np.array_equal(dev, want_dev)
    for buf in (qb, kb, vb, codes, scales):
        be.free(buf)


@pytest.mark.parametrize("s_q,heads", [(140, 2), (256, 80)])  # keys mode, rows mode
def test_output_on_a_16_byte_boundary(backend, s_q, heads):
    """The output rows leave as 32-byte stores when they start on 32 bytes, as 16-byte ones otherwise: the same bits."""
    from thinfer_b200 import _lib as L

    be, n = backend, s_q * heads * 128 * 2
    q, k, v = _inputs(1, s_q, 150, heads, heads, 99)
    want = _run(be, q, k, v, SCALE)
    qb, kb, vb, out = be.upload(q), be.upload(k), be.upload(v), be.upload(np.full(n // 2 + 16, 0x7FC0, np.uint16))
    be.scope().sdpa(qb, kb, vb, L.Buf(out.id, 16, n), 1, s_q, 150, heads, heads, SCALE)
    be.submit(30000)
    got = be.read_buffer(out, np.uint16)
    assert np.array_equal(got[8: 8 + n // 2], want.ravel())
    assert (got[:8] == 0x7FC0).all() and (got[8 + n // 2:] == 0x7FC0).all()
    for buf in (qb, kb, vb, out):
        be.free(buf)
