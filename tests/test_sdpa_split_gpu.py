"""Attention with few blocks of 128 query rows and many keys: clusters of 2 to 8 CTAs share a block's key tiles (sdpa_split in
csrc/rules.h; its rule is tested in test_rules.py). Against the restated reference, same tolerance and reason as test_sdpa_gpu.py."""
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
from conftest import ROOT, dev_scales_to_canonical, rel_fro
from test_sdpa_gpu import TOL, _inputs, _run

pytestmark = pytest.mark.gpu
SCALE = float(1.0 / np.sqrt(128.0))


@pytest.mark.parametrize("b,s_q,s_k,h_q,h_kv,spread", [
    (1, 128, 2048, 1, 1, 1.0),    # one block, 16 tiles: eight CTAs of two
    (1, 1, 2000, 3, 1, 1.0),      # one row; a ragged last tile; grouped heads
    (1, 300, 1700, 4, 2, 6.0),    # 12 blocks of which a third have 44 rows, 14 tiles in uneven shares, peaked rows
    (2, 200, 1300, 4, 4, 1.0),    # 16 blocks, two batches: rows past a sequence's end belong to the next one
    (1, 700, 2305, 4, 4, 1.0),    # 24 blocks, 19 tiles, one key in the last
    (1, 520, 1540, 6, 6, 1.0),    # 30 blocks, 13 tiles
    (1, 1280, 1700, 7, 7, 1.0),   # 70 blocks: two CTAs each
    (1, 260, 1025, 2, 2, 1.0),    # 9 tiles
])
def test_split_matches_reference_recurrence(backend, b, s_q, s_k, h_q, h_kv, spread):
    q, k, v = _inputs(b, s_q, s_k, h_q, h_kv, 17 * s_q + s_k, spread)
    got = O.bf16_to_f32(_run(backend, q, k, v, SCALE))
    want = O.bf16_to_f32(O.ref_sdpa(q, k, v, SCALE))
    assert not np.isnan(got).any()
    for bi in range(b):
        for h in range(h_q):
            for r in range(0, s_q, 128):  # per block: an error in one cluster must not hide in the norm over all of them
                assert rel_fro(got[bi, r: r + 128, h], want[bi, r: r + 128, h]) <= 1.5 * TOL, (bi, h, r)
    assert rel_fro(got, want) <= TOL


FIRST_CALLS = """
import threading
import numpy as np
import thinfer_b200 as T
s_q, s_k, heads, n = 200, 2048, 2, 8
rng = np.random.default_rng(5)
q, k, v = (rng.standard_normal((1, s, heads, 128)).astype(np.float32) for s in (s_q, s_k, s_k))
q, k, v = ((t.view(np.uint32) >> 16).astype(np.uint16) for t in (q, k, v))
backends = [T.Backend(0) for _ in range(n)]
bufs = [[be.upload(t) for t in (q, k, v)] + [be.allocate(q.nbytes)] for be in backends]
gate, got = threading.Barrier(n), [None] * n
def call(i):
    gate.wait()
    backends[i].scope().sdpa(*bufs[i], 1, s_q, s_k, heads, heads, 0.088)
    backends[i].submit(30000)
    got[i] = backends[i].read_buffer(bufs[i][3], np.uint16)
threads = [threading.Thread(target=call, args=(i,)) for i in range(n)]
[t.start() for t in threads]
[t.join() for t in threads]
assert all(g is not None and np.array_equal(g, got[0]) for g in got), [g is not None and int((g != got[0]).sum()) for g in got]
"""


def test_first_calls_of_several_threads():
    """The first calls of a process, all at once on contexts of their own, take the same kernel: the same bits."""
    for _ in range(3):
        subprocess.run([sys.executable, "-c", FIRST_CALLS], check=True, cwd=ROOT, timeout=300)


@pytest.mark.parametrize("jumps", [
    {0: 400.0},                                        # the first share's maximum is far above the others'
    {2047: 900.0},                                     # the last key's: every other share underflows
    {300: 12.0, 700: 24.0, 1100: 300.0, 1900: 600.0},  # every few shares a larger one
    {j: -np.inf for j in range(256, 1024)},            # shares without a key that weighs anything
])
def test_shares_of_different_size(backend, jumps):
    """Score of key j (exp2 domain) = jumps[j], small noise elsewhere, the same for every row."""
    s_q, s_k, heads, d = 200, 2048, 2, 128
    k = np.zeros((1, s_k, heads, d), np.float32)
    rng = np.random.default_rng(3)
    k[..., 0] = rng.uniform(-1, 1, (1, s_k, heads))
    for j, x in jumps.items():
        k[:, j, :, 0] = x
    q = np.zeros((1, s_q, heads, d), np.float32)
    q[..., 0] = np.log(2.0) / SCALE
    v = rng.standard_normal((1, s_k, heads, d)).astype(np.float32)
    live = [j for j in range(s_k) if jumps.get(j, 0.0) != -np.inf]  # the reference's recurrence has no key without weight
    q, k, v = (O.f32_to_bf16(t) for t in (q, k, v))
    got = O.bf16_to_f32(_run(backend, q, k, v, SCALE))
    want = O.bf16_to_f32(O.ref_sdpa(q, np.ascontiguousarray(k[:, live]), np.ascontiguousarray(v[:, live]), SCALE))
    assert not np.isnan(got).any() and rel_fro(got, want) <= TOL


@pytest.mark.parametrize("s_q,heads,s_k,offset", [(200, 2, 2048, 0), (300, 8, 1300, 16)])
def test_split_outputs(backend, s_q, heads, s_k, offset):
    """The NVFP4 copy equals the quantiser's on the bf16 output, whose rows may start on 16 bytes."""
    from thinfer_b200 import _lib as L

    be, cols = backend, heads * 128
    q, k, v = _inputs(1, s_q, s_k, heads, heads, 512)
    plain = _run(be, q, k, v, SCALE).reshape(s_q, cols)
    g = O.global_scale(O.amax_bf16(plain))
    qb, kb, vb = be.upload(q), be.upload(k), be.upload(v)
    want_c, want_s = O.quantize_act(plain, g)
    want_dev = O.scales_to_device_layout(want_s)
    codes, scales, n = be.allocate(s_q * cols // 2), be.upload(np.full(want_dev.size, 0x7F, np.uint8)), s_q * cols * 2
    out = be.upload(np.full(n // 2 + 16, 0x7FC0, np.uint16))
    be.scope().sdpa(qb, kb, vb, L.Buf(out.id, offset, n), 1, s_q, s_k, heads, heads, SCALE, out_nvfp4=(codes, scales, g))
    be.submit(30000)
    got = be.read_buffer(out, np.uint16)
    assert np.array_equal(got[offset // 2: offset // 2 + n // 2].reshape(s_q, cols), plain)
    assert (got[: offset // 2] == 0x7FC0).all() and (got[offset // 2 + n // 2:] == 0x7FC0).all()
    assert np.array_equal(be.read_buffer(codes).reshape(s_q, cols // 2), want_c)
    dev = be.read_buffer(scales)
    assert np.array_equal(dev_scales_to_canonical(dev, s_q, cols), want_s) and np.array_equal(dev, want_dev)
    for buf in (qb, kb, vb, out, codes, scales):
        be.free(buf)
