"""The CTA-pair kernel's epilogues: one kernel for plain and GELU outputs, one with a gated residual (which arrives by TMA in the buffer
that the result replaces it in), one with the NVFP4 copy and one with SwiGLU, and the general one that a long K and many tiles get.
Every output element is compared, bit for bit, with the same rows computed about 100 at a time by the 1-CTA kernel, whose epilogue
arithmetic is the same and whose sums run over K in the same order."""
import numpy as np
import pytest

import oracle as O
from conftest import dev_scales_to_canonical

pytestmark = pytest.mark.gpu

SHAPES = [
    (2100, 2312, 320),   # 90 tiles; 8 columns in the last column tile, 52 rows in the last row tile
    (2305, 4648, 64),    # 190 tiles, three of a pair; one row in the last row tile, 40 columns in the last column tile
    (4400, 2304, 3104),  # 162 tiles, K past the limits of the plain and the NVFP4 output's own epilogue
    (4400, 2304, 3616),  # ... and of GELU's
    (257, 19200, 256),   # 150 tiles: the last two as halves of 128 columns
]


def _slices(m):
    step = next(s for s in range(96, 129) if m % s == 0 or m % s > 16)  # 17 rows and more: up to 16 take a kernel that rounds alpha and bias apart
    return [(r, min(step, m - r)) for r in range(0, m, step)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("kind", ["plain", "gelu", "chain", "gate", "gelu_gate", "gate_in_place", "swiglu", "window"])
def test_bf16_outputs(backend, m, n, k, kind):
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    if kind == "swiglu":
        n = n // 16 * 16
    be, rng, g = backend, np.random.default_rng(m + n + k), 0.002
    a = O.f32_to_bf16(rng.standard_normal((m, k), np.float32))
    W = T.Nvfp4Weight.from_dense(be, rng.standard_normal((n, k), np.float32) * np.float32(0.02), O.f32_to_bf16(rng.standard_normal(n, np.float32)))
    gated = "gate" in kind
    res = O.f32_to_bf16(rng.standard_normal((m, n), np.float32))
    cols = n // 2 if kind == "swiglu" else n
    ldo, off = (n + 24, 8) if kind == "window" else (cols, 0)
    ab, gb, rb = be.upload(a), be.upload(O.f32_to_bf16(rng.standard_normal(n, np.float32))), be.upload(res)
    out, part = be.upload(np.full((m + 1, ldo), 0x7FC0, np.uint16)), be.upload(np.full((m, ldo), 0x7FC0, np.uint16))
    kw = dict(act=L.ACT_GELU_TANH if "gelu" in kind else L.ACT_NONE, chain=kind == "chain", swiglu=kind == "swiglu")
    if kind == "window":
        kw.update(n_offset=off, ldo=ldo)
    if kind == "gate_in_place":
        be.write_buffer(out, res)
    sc = be.scope()
    sc.linear(ab, m, W, g, out, gate=gb if gated else None, residual=(out if kind == "gate_in_place" else rb) if gated else None, **kw)
    for r, rows in _slices(m):
        view = lambda buf, c: L.Buf(buf.id, r * c * 2, rows * c * 2)
        sc.linear(view(ab, k), rows, W, g, view(part, ldo), gate=gb if gated else None, residual=view(rb, n) if gated else None, **kw)
    be.submit(30000)
    got, want = be.read_buffer(out, np.uint16).reshape(m + 1, ldo), be.read_buffer(part, np.uint16).reshape(m, ldo)
    assert (got[m] == 0x7FC0).all()  # nothing is written past the last row ...
    assert np.array_equal(got[:m], want)  # ... or outside the window
    W.free(be)
    for buf in (ab, gb, rb, out, part):
        be.free(buf)


@pytest.mark.parametrize("m,n,k", [(2100, 2368, 320), (2305, 4672, 64), (4400, 2304, 3104), (257, 18944, 256)])
@pytest.mark.parametrize("act,offset,bf16", [(0, 0, False), (1, 0, False), (1, 16, False), (1, 0, True)])
def test_nvfp4_output(backend, m, n, k, act, offset, bf16):
    """Codes and scales of the fused NVFP4 copy; also into a buffer that starts on 16 bytes only, and with the bf16 output as well."""
    import thinfer_b200 as T
    from thinfer_b200.backend import device_scales_bytes
    from thinfer_b200 import _lib as L

    be, rng, g, gq = backend, np.random.default_rng(m + n + k), 0.002, 0.003
    W = T.Nvfp4Weight.from_dense(be, rng.standard_normal((n, k), np.float32) * np.float32(0.02), O.f32_to_bf16(rng.standard_normal(n, np.float32)))
    ab = be.upload(O.f32_to_bf16(rng.standard_normal((m, k), np.float32)))
    codes, scales, out, part = be.allocate(m * n // 2 + 16), be.allocate(device_scales_bytes(m, n)), be.allocate(m * n * 2), be.allocate(m * n * 2)
    sc = be.scope()
    sc.linear(ab, m, W, g, out if bf16 else None, act=act, out_nvfp4=(L.Buf(codes.id, offset, m * n // 2), scales, gq))
    for r, rows in _slices(m):
        sc.linear(L.Buf(ab.id, r * k * 2, rows * k * 2), rows, W, g, L.Buf(part.id, r * n * 2, rows * n * 2), act=act)
    qc, qs, _ = sc.act_quant(part, m, n, gq, device_layout=True)
    be.submit(30000)
    assert np.array_equal(be.read_buffer(codes, np.uint8, count=m * n // 2, offset=offset), be.read_buffer(qc))
    assert np.array_equal(dev_scales_to_canonical(be.read_buffer(scales), m, n), dev_scales_to_canonical(be.read_buffer(qs), m, n))
    if bf16:
        assert np.array_equal(be.read_buffer(out, np.uint16), be.read_buffer(part, np.uint16))
    W.free(be)
    for buf in (ab, codes, scales, out, part, qc, qs):
        be.free(buf)
