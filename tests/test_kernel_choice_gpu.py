"""Which kernel a linear takes must not show in its bits: shapes on both sides of the rules (one wave of 128-wide tiles, two with a
short K, pairs working on halves of their tiles in the only wave), every epilogue, against the same rows computed about 100 at a time
(1-CTA kernel, few tiles), and against the oracle."""
import numpy as np
import pytest

import oracle as O
from conftest import dev_scales_to_canonical, rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [
    (700, 3072, 512),    # 144 tiles of 128 x 128: one wave
    (300, 6144, 288),    # 144, ragged rows and K
    (769, 3072, 2048),   # 168: two waves, single CTAs where there is no gated residual
    (513, 4096, 800),    # 160 tiles, the same
    (513, 4096, 768),    # ... and pairs for a shorter K
    (769, 3072, 2080),   # the same with K past the limit: 48 tiles of 256 x 256 on pairs
    (513, 3200, 2112),   # 3 x 13 pair tiles, a ragged column tile: not halved
    (1280, 2048, 2304),  # 40 pair tiles: not halved (more halves than pairs)
    (130, 9472, 64),     # 148 tiles: exactly one wave
    (130, 9600, 2304),   # 150: pairs, 38 tiles, ragged column tile
])
@pytest.mark.parametrize("kind", ["plain", "gelu", "gate", "chain"])
def test_kernel_choice_does_not_show(backend, m, n, k, kind):
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    be, rng, g = backend, np.random.default_rng(m + n + k), 0.002
    a = O.f32_to_bf16(rng.standard_normal((m, k), np.float32))
    w, bias = rng.standard_normal((n, k), np.float32) * np.float32(0.02), O.f32_to_bf16(rng.standard_normal(n, np.float32))
    W = T.Nvfp4Weight.from_dense(be, w, bias)
    gate, res = O.f32_to_bf16(rng.standard_normal(n, np.float32)), O.f32_to_bf16(rng.standard_normal((m, n), np.float32))
    gated = kind in ("gate", "chain")
    ab, gb, rb = be.upload(a), be.upload(gate), be.upload(res)
    out, part = be.upload(np.full((m, n), 0x7FC0, np.uint16)), be.allocate(m * n * 2)
    kw = dict(act=L.ACT_GELU_TANH if kind in ("gelu", "chain") else L.ACT_NONE, chain=kind == "chain")
    sc = be.scope()
    sc.linear(ab, m, W, g, out, gate=gb if gated else None, residual=rb if gated else None, **kw)
    # slices of 17 rows and more: the skinny kernel (up to 16) rounds the products with alpha before it adds the bias
    step = 96 if m % 96 > 16 else 100
    for r in range(0, m, step):
        rows = min(step, m - r)
        assert rows > 16
        view = lambda buf, cols: L.Buf(buf.id, r * cols * 2, rows * cols * 2)
        sc.linear(view(ab, k), rows, W, g, view(part, n), gate=gb if gated else None, residual=view(rb, n) if gated else None, **kw)
    be.submit(30000)
    got, want = be.read_buffer(out, np.uint16).reshape(m, n), be.read_buffer(part, np.uint16).reshape(m, n)
    assert np.array_equal(got, want)
    if kind == "plain":
        wc, ws, gw = O.quantize_weight(w)
        rows = np.r_[0:3, m // 2: m // 2 + 3, m - 3: m]
        ref = O.bf16_to_f32(O.linear(a[rows], g, wc, ws, gw, bias=bias))
        assert rel_fro(O.bf16_to_f32(got[rows]), ref) <= 1e-3
    W.free(be)
    for buf in (ab, gb, rb, out, part):
        be.free(buf)


@pytest.mark.parametrize("m,n,k", [(200, 512, 256), (640, 1024, 544), (257, 2304, 256)])  # 2, 12 and 18 pair tiles, all in halves
def test_halves_in_the_only_wave(backend, m, n, k):
    """The dense arm runs on the pair kernel whatever the size: its only wave in halves. Beside it, on the 1-CTA kernel: the NVFP4
    output, the bf16 output of the kernel that makes it, and SwiGLU."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L
    from thinfer_b200.backend import device_scales_bytes

    be, rng, g = backend, np.random.default_rng(m), 0.002
    a = O.f32_to_bf16(rng.standard_normal((m, k), np.float32))
    W = T.Nvfp4Weight.from_dense(be, rng.standard_normal((n, k), np.float32) * np.float32(0.02))
    W.prepare_dense(be)
    ab, y, codes, scales = be.upload(a), be.allocate(m * n * 2), be.allocate(m * n // 2), be.allocate(device_scales_bytes(m, n))
    sw, dense = be.allocate(m * n), be.allocate(m * n * 2)
    sc = be.scope()
    sc.linear(ab, m, W, g, y)
    y2 = be.allocate(m * n * 2)
    sc.linear(ab, m, W, g, y2, out_nvfp4=(codes, scales, 0.001))
    sc.linear(ab, m, W, g, sw, swiglu=True)
    sc.linear(ab, m, W, g, dense, dense_act=True)
    be.submit(30000)
    yv = be.read_buffer(y, np.uint16).reshape(m, n)
    assert np.array_equal(be.read_buffer(y2, np.uint16).reshape(m, n), yv)
    oc, os_ = O.quantize_act(yv, 0.001)
    assert np.array_equal(be.read_buffer(codes).reshape(m, n // 2), oc)
    assert np.array_equal(dev_scales_to_canonical(be.read_buffer(scales), m, n), os_)  # the GEMM leaves the rows past m alone
    f = O.bf16_to_f32(yv).astype(np.float64)
    want = f[:, 0::2] / (1.0 + np.exp(-f[:, 0::2])) * f[:, 1::2]
    assert rel_fro(O.bf16_to_f32(be.read_buffer(sw, np.uint16)).reshape(m, n // 2), want) <= 8e-3  # from bf16-rounded inputs: 2 x 2^-9 and the output's
    d = be.read_buffer(dense, np.uint16)
    img = O.bf16_to_f32(be.read_buffer(W.dense, np.uint16)).reshape(n, k).astype(np.float64)
    ref = O.bf16_to_f32(a).astype(np.float64) @ img.T * W.global_scale
    assert rel_fro(O.bf16_to_f32(d).reshape(m, n), ref) <= 4e-3  # one bf16 rounding: 2^-9 at most
    W.free(be)
    for buf in (ab, y, y2, codes, scales, sw, dense):
        be.free(buf)


@pytest.mark.parametrize("m,n,k", [
    (1, 512, 256), (200, 512, 256),  # 64-wide tiles
    (100, 9600, 64),                 # 128-wide: 75 tiles
    (300, 6144, 288),                # 144 tiles, the last rows ragged
    (130, 9408, 96),                 # the last tile 64 columns wide
    (40, 37888, 96),                 # 256-wide: 148 tiles
])
@pytest.mark.parametrize("act,chain,keep_bf16", [(0, False, True), (1, False, False), (1, True, True), (0, True, False)])
def test_nvfp4_output_of_the_one_cta_kernel(backend, m, n, k, act, chain, keep_bf16):
    """Codes and scales of the fused output quantiser, in a window of a wider operand, against the oracle quantiser on the bf16
    output of the same linear; nothing else in the operand is touched."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L
    from thinfer_b200.backend import device_scales_bytes

    be, rng, g, off, ldo = backend, np.random.default_rng(m + n), 0.002, 64, n + 192
    ab = be.upload(O.f32_to_bf16(rng.standard_normal((m, k), np.float32)))
    W = T.Nvfp4Weight.from_dense(be, rng.standard_normal((n, k), np.float32) * np.float32(0.05), O.f32_to_bf16(rng.standard_normal(n, np.float32)))
    plain, wide = be.allocate(m * n * 2), be.upload(np.full((m, ldo), 0x7FC0, np.uint16))
    codes, scales = be.upload(np.full((m, ldo // 2), 0xA5, np.uint8)), be.upload(np.full(device_scales_bytes(m, ldo), 0x55, np.uint8))
    sc, go = be.scope(), 0.0007
    sc.linear(ab, m, W, g, wide if keep_bf16 else None, act=act, chain=chain, n_offset=off, ldo=ldo, out_nvfp4=(codes, scales, go))
    if m <= 16:
        sc.act_quant_shared(ab, m, k, g)  # not the skinny kernel, which rounds alpha and bias apart
    sc.linear(ab, m, W, g, plain, act=act, chain=chain, flags=L.LINEAR_A_PREQUANTIZED if m <= 16 else 0)
    be.submit(30000)
    y = be.read_buffer(plain, np.uint16).reshape(m, n)
    oc, os_ = O.quantize_act(y, go)
    c = be.read_buffer(codes).reshape(m, ldo // 2)
    assert np.array_equal(c[:, off // 2: (off + n) // 2], oc)
    assert (c[:, : off // 2] == 0xA5).all() and (c[:, (off + n) // 2:] == 0xA5).all()
    s = dev_scales_to_canonical(be.read_buffer(scales), m, ldo)
    assert np.array_equal(s[:, off // 16: (off + n) // 16], os_)
    assert (s[:, : off // 16] == 0x55).all() and (s[:, (off + n) // 16:] == 0x55).all()
    b = be.read_buffer(wide, np.uint16).reshape(m, ldo)
    assert np.array_equal(b[:, off: off + n], y) if keep_bf16 else (b == 0x7FC0).all()
    assert (b[:, :off] == 0x7FC0).all() and (b[:, off + n:] == 0x7FC0).all()
    W.free(be)
    for buf in (ab, plain, wide, codes, scales):
        be.free(buf)


@pytest.mark.parametrize("m,n,k,chain", [(1600, 4096, 512, False), (1600, 4112, 96, True), (2048, 9472, 64, False)])
def test_swiglu_of_either_kernel(backend, m, n, k, chain):
    """Rows on the pair kernel and the same rows a hundred at a time on the 1-CTA kernel (64-wide and 128-wide tiles, ragged columns)."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    be, rng, g, cols = backend, np.random.default_rng(n), 0.002, n // 2
    ab = be.upload(O.f32_to_bf16(rng.standard_normal((m, k), np.float32)))
    W = T.Nvfp4Weight.from_dense(be, rng.standard_normal((n, k), np.float32) * np.float32(0.1), O.f32_to_bf16(rng.standard_normal(n, np.float32)))
    out, part = be.allocate(m * cols * 2), be.upload(np.full((m, cols + 24), 0x7FC0, np.uint16))
    sc = be.scope()
    sc.linear(ab, m, W, g, out, swiglu=True, chain=chain)
    for r in range(0, m, 100):
        rows = min(100, m - r)
        sc.linear(L.Buf(ab.id, r * k * 2, rows * k * 2), rows, W, g, L.Buf(part.id, r * (cols + 24) * 2, rows * (cols + 24) * 2), swiglu=True,
                  chain=chain, n_offset=8, ldo=cols + 24)
    be.submit(30000)
    got, want = be.read_buffer(part, np.uint16).reshape(m, cols + 24), be.read_buffer(out, np.uint16).reshape(m, cols)
    assert np.array_equal(got[:, 8: 8 + cols], want)
    assert (got[:, :8] == 0x7FC0).all() and (got[:, 8 + cols:] == 0x7FC0).all()
    W.free(be)
    for buf in (ab, out, part):
        be.free(buf)


@pytest.mark.parametrize("m,n,k,forms", [
    (18944, 64, 96, ("plain", "quant", "swiglu")),   # 148 row tiles of a W of less than one scale block
    (18817, 128, 64, ("plain", "quant", "swiglu")),  # the same, a whole block
    (256, 18704, 96, ("plain", "swiglu")),           # 256-wide tiles, the last with 16 columns
    (129, 18816, 288, ("plain", "quant")),           # ... with 128: one whole scale block of two
    (512, 9280, 96, ("plain", "quant")),
    (40, 37760, 96, ("plain", "quant", "swiglu")),
])
def test_last_tile_of_less_than_one_scale_block(backend, m, n, k, forms):
    """256-wide tiles of the 1-CTA kernel whose last one needs one of two blocks of W's scales: the same rows in slices, and the
    oracle."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L
    from thinfer_b200.backend import device_scales_bytes

    be, rng, g, go = backend, np.random.default_rng(m + n), 0.002, 0.0007
    a = O.f32_to_bf16(rng.standard_normal((m, k), np.float32))
    w, bias = rng.standard_normal((n, k), np.float32) * np.float32(0.1), O.f32_to_bf16(rng.standard_normal(n, np.float32))
    W = T.Nvfp4Weight.from_dense(be, w, bias)
    ab, out, part = be.upload(a), be.allocate(m * n * 2), be.allocate(m * n * 2)
    sc = be.scope()
    sc.linear(ab, m, W, g, out)
    step = 1024 if n < 256 else 24 if m < 100 else 96
    for r in range(0, m, step):  # 64- and 128-wide tiles
        rows = min(step, m - r)
        if rows <= 16:
            continue  # the skinny kernel rounds the products with alpha before it adds the bias
        sc.linear(L.Buf(ab.id, r * k * 2, rows * k * 2), rows, W, g, L.Buf(part.id, r * n * 2, rows * n * 2))
    be.submit(30000)
    y, want = be.read_buffer(out, np.uint16).reshape(m, n), be.read_buffer(part, np.uint16).reshape(m, n)
    whole = m - (m % step if m % step <= 16 else 0)
    assert np.array_equal(y[:whole], want[:whole])
    rows = np.r_[0:3, m - 3: m]
    wc, ws, gw = O.quantize_weight(w)
    assert rel_fro(O.bf16_to_f32(y[rows]), O.bf16_to_f32(O.linear(a[rows], g, wc, ws, gw, bias=bias))) <= 1e-3
    bufs = [ab, out, part]
    if "quant" in forms:
        codes, scales = be.allocate(m * n // 2), be.allocate(device_scales_bytes(m, n))
        sc.linear(ab, m, W, g, None, out_nvfp4=(codes, scales, go))
        be.submit(30000)
        oc, os_ = O.quantize_act(y, go)
        assert np.array_equal(be.read_buffer(codes).reshape(m, n // 2), oc)
        assert np.array_equal(dev_scales_to_canonical(be.read_buffer(scales), m, n), os_)
        bufs += [codes, scales]
    if "swiglu" in forms:
        sw = be.allocate(m * n)
        sc.linear(ab, m, W, g, sw, swiglu=True)
        be.submit(30000)
        f = O.bf16_to_f32(y).astype(np.float64)
        want = f[:, 0::2] / (1.0 + np.exp(-f[:, 0::2])) * f[:, 1::2]
        assert rel_fro(O.bf16_to_f32(be.read_buffer(sw, np.uint16)).reshape(m, n // 2), want) <= 8e-3  # from bf16-rounded inputs: 2 x 2^-9 and the output's
        bufs.append(sw)
    W.free(be)
    for buf in bufs:
        be.free(buf)


@pytest.mark.parametrize("budget", [False, True])
@pytest.mark.parametrize("n,k", [(2048, 8192), (3648, 2080), (4096, 96)])
def test_few_rows_in_a_scratch_full_of_others(n, k, budget):
    """Few rows of activations whose tensor map reaches over the scratch behind them: what an earlier call has left there must not
    show. With a budget that has no byte to spare the scratch is as large as the operand and the map ends with it."""
    import thinfer_b200 as T
    from thinfer_b200.backend import device_scales_bytes

    rng, g, go = np.random.default_rng(k), 0.002, 0.0007
    big, few = 120, (17, 20, 31)
    a = O.f32_to_bf16(rng.standard_normal((big, k), np.float32))
    w = rng.standard_normal((n, k), np.float32) * np.float32(0.05)
    size = lambda m: m * n * 2
    fixed = 4 * size(big) + (160 << 20)  # room for the f32 weight while it is quantised
    be = T.Backend(0, fixed if budget else 0)
    try:
        W = T.Nvfp4Weight.from_dense(be, w, O.f32_to_bf16(rng.standard_normal(n, np.float32)))
        ab, sc = be.upload(a), be.scope()
        outs = [be.upload(np.full((big, n), 0x7FC0, np.uint16)) for _ in range(2)]
        sw, codes, scales = be.allocate(size(big) // 2), be.allocate(big * n // 2), be.allocate(device_scales_bytes(big, n))
        if budget:  # the scratch of 17 rows is the last that fits
            live = sum(v for key, v in be.mem_snapshot().items() if key.startswith("live"))
            filler = be.allocate(fixed - live - (17 * k // 2 + device_scales_bytes(17, k)))
            sc.linear(ab, 17, W, g, outs[0])
            be.submit(30000)
            be.free(filler)
            be.write_buffer(outs[0], np.full((big, n), 0x7FC0, np.uint16))
        sc.linear(ab, big, W, g, outs[1])
        be.submit(30000)
        want = be.read_buffer(outs[1], np.uint16).reshape(big, n)
        for m in few:
            sc.linear(ab, m, W, g, outs[0])
            sc.linear(ab, m, W, g, sw, swiglu=True)
            sc.linear(ab, m, W, g, None, out_nvfp4=(codes, scales, go))
            be.submit(30000)
            got = be.read_buffer(outs[0], np.uint16).reshape(big, n)
            assert np.array_equal(got[:m], want[:m])
            assert (got[m:] == 0x7FC0).all()
            oc, os_ = O.quantize_act(want[:m], go)
            assert np.array_equal(be.read_buffer(codes)[: m * n // 2].reshape(m, n // 2), oc)
            assert np.array_equal(dev_scales_to_canonical(be.read_buffer(scales), m, n), os_)
            f = O.bf16_to_f32(want[:m]).astype(np.float64)
            ref = f[:, 0::2] / (1.0 + np.exp(-f[:, 0::2])) * f[:, 1::2]
            assert rel_fro(O.bf16_to_f32(be.read_buffer(sw, np.uint16))[: m * n // 2].reshape(m, n // 2), ref) <= 8e-3  # from bf16-rounded inputs
            be.write_buffer(outs[0], np.full((big, n), 0x7FC0, np.uint16))
    finally:
        be.close()
