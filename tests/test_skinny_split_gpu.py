"""Linears of up to 16 rows whose K tiles are shared by a cluster of CTAs (skinny_split_rule in csrc/rules.h, tested in test_rules.py),
against the oracle: relative Frobenius error <= 1e-3, as for every linear; in fact the products are exact and only the order of
the f32 sums differs."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_fro

pytestmark = pytest.mark.gpu


def _problem(m, n, k, seed):
    a = O.f32_to_bf16(O.gaussian(m * k, 0xA100 + seed).reshape(m, k))
    w = (O.gaussian(n * k, 0xB100 + seed) * np.float32(0.02)).reshape(n, k)
    return a, O.quantize_weight(w), O.f32_to_bf16(O.gaussian(n, 0xC100 + seed) * np.float32(0.01))


@pytest.mark.parametrize("m,n,k", [
    (1, 3072, 3072),    # four CTAs of three K tiles
    (1, 264, 14336),    # eight CTAs; 8 columns in the last tile; K past what the kernel without clusters can hold
    (3, 1000, 4128),    # 17 K tiles, the last of 32 elements, in uneven shares
    (4, 4736, 6144),    # 37 tiles
    (5, 3072, 3072),    # more than four rows: 512 threads
    (16, 9216, 6176),   # two CTAs, 25 K tiles
    (16, 136, 1024),    # four K tiles
    (7, 2304, 9216),
])
@pytest.mark.parametrize("mode", ["plain", "gelu", "gate", "chain", "window"])
def test_epilogues(backend, m, n, k, mode):
    import thinfer_b200 as T

    be = backend
    a, (wc, ws, gw), b = _problem(m, n, k, m + n)
    ga = O.global_scale(O.amax_bf16(a))
    W = T.Nvfp4Weight.from_packed(be, wc, ws, gw, b)
    gate, res = O.f32_to_bf16(O.gaussian(n, 0xD000)), O.f32_to_bf16(O.gaussian(m * n, 0xE000).reshape(m, n))
    ldo, off = (n + 24, 8) if mode == "window" else (n, 0)
    ab, gb, rb, out = be.upload(a), be.upload(gate), be.upload(res), be.upload(np.full((m + 1, ldo), 0x7FC0, np.uint16))
    kw, okw = {}, {}
    if mode in ("gelu", "chain"):
        kw["act"] = okw["act"] = 1
    if mode in ("gate", "chain"):
        kw.update(gate=gb, residual=rb)
        okw.update(gate=gate, residual=res)
    if mode == "chain":
        kw["chain"] = okw["chain"] = True
    if mode == "window":
        kw.update(n_offset=off, ldo=ldo)
    for _ in range(3):  # the words that the cluster shares are those of the launch
        be.scope().linear(ab, m, W, ga, out, **kw)
    be.submit(30000)
    got = be.read_buffer(out, np.uint16).reshape(m + 1, ldo)
    want = O.bf16_to_f32(O.linear(a, ga, wc, ws, gw, bias=b, **okw))
    assert rel_fro(O.bf16_to_f32(got[:m, off: off + n]), want) <= 1e-3
    for i in range(m):  # a row lost in one CTA must not hide in the norm over all
        assert rel_fro(O.bf16_to_f32(got[i, off: off + n]), want[i]) <= 2e-3
    assert (got[m] == 0x7FC0).all() and (got[:m, :off] == 0x7FC0).all() and (got[:m, off + n:] == 0x7FC0).all()
    W.free(be)
    for buf in (ab, gb, rb, out):
        be.free(buf)


@pytest.mark.parametrize("m,n,k", [(1, 272, 14336), (2, 9216, 3072), (3, 1008, 4128), (5, 3072, 3072), (16, 144, 1024), (16, 6144, 6176)])
@pytest.mark.parametrize("chain", [False, True])
def test_swiglu(backend, m, n, k, chain):
    """Against the GEMM's epilogue, which takes over where the scratch is filled beforehand: the f32 sums differ in their order only, so that
    few results are another bf16 value (2^-8 of them at most)."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    be = backend
    a, (wc, ws, gw), b = _problem(m, n, k, m + n)
    ga = O.global_scale(O.amax_bf16(a))
    W = T.Nvfp4Weight.from_packed(be, wc, ws, gw, b)
    ldo, off = n // 2 + 24, 8
    ab, got = be.upload(a), []
    for flags in (L.LINEAR_A_PREQUANTIZED, 0):
        out = be.upload(np.full((m + 1, ldo), 0x7FC0, np.uint16))
        sc = be.scope()
        sc.act_quant_shared(ab, m, k, ga)
        sc.linear(ab if flags == 0 else None, m, W, ga, out, flags=flags, swiglu=True, chain=chain, n_offset=off, ldo=ldo)
        be.submit(30000)
        got.append(be.read_buffer(out, np.uint16).reshape(m + 1, ldo))
        be.free(out)
    want, have = (O.bf16_to_f32(g[:m, off: off + n // 2]) for g in got)
    for i in range(m):
        assert rel_fro(have[i], want[i]) <= (4e-3 if chain else 1e-3)  # chain: halves of the pair rounded to bf16 before, 2^-8 where they fall the other way
    assert (got[1][m] == 0x7FC0).all() and (got[1][:m, :off] == 0x7FC0).all() and (got[1][:m, off + n // 2:] == 0x7FC0).all()
    W.free(be)
    be.free(ab)


@pytest.mark.parametrize("m,n,k", [(16, 1024, 4128), (5, 264, 6144)])
def test_scratch_holds_the_activations(backend, m, n, k):
    """A call that would have run the quantiser leaves what the quantiser leaves: the shared scratch serves the next call."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    be = backend
    a, (wc, ws, gw), _ = _problem(m, n, k, 5)
    assert m * k > 24576
    ga = O.global_scale(O.amax_bf16(a))
    W = T.Nvfp4Weight.from_packed(be, wc, ws, gw, None)
    ab, other, out, ref = be.upload(a), be.upload(np.roll(a, 1)), be.allocate(m * n * 2), be.allocate(m * n * 2)
    sc = be.scope()
    sc.act_quant_shared(ab, m, k, ga)
    sc.linear(None, m, W, ga, ref, flags=L.LINEAR_A_PREQUANTIZED)
    sc.act_quant_shared(other, m, k, ga)
    sc.linear(ab, m, W, ga, out)
    sc.linear(None, m, W, ga, out, flags=L.LINEAR_A_PREQUANTIZED)
    be.submit(30000)
    assert np.array_equal(be.read_buffer(out, np.uint16), be.read_buffer(ref, np.uint16))
    W.free(be)
    for buf in (ab, other, out, ref):
        be.free(buf)


@pytest.mark.parametrize("flaw", ["window", "weight", "bias"])
@pytest.mark.parametrize("swiglu", [False, True])
def test_refused_call_leaves_its_own_activations(backend, flaw, swiglu):
    """The quantiser runs ahead of a linear's other checks: after a refused call the scratch holds that call's activations, not an earlier
    call's under the same shape."""
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L
    from thinfer_b200.backend import InvalidArgument

    be, (m, n, k) = backend, (16, 1024, 4128)
    a, (wc, ws, gw), b = _problem(m, n, k, 13)
    ga, cols = O.global_scale(O.amax_bf16(a)), n // 2 if swiglu else n
    W = T.Nvfp4Weight.from_packed(be, wc, ws, gw, b)
    ab, other, out, ref = be.upload(a), be.upload(np.roll(a, 1)), be.allocate(m * cols * 2), be.allocate(m * cols * 2)
    sc = be.scope()
    sc.act_quant_shared(ab, m, k, ga)
    sc.linear(None, m, W, ga, ref, flags=L.LINEAR_A_PREQUANTIZED, swiglu=swiglu)
    sc.act_quant_shared(other, m, k, ga)
    V = T.Nvfp4Weight(n, k, W.codes, W.scales_device, gw, W.bias)
    if flaw == "weight":
        V.codes = L.Buf(W.codes.id, 0, n * k // 2 - 16)
    if flaw == "bias":
        V.bias = L.Buf(W.bias.id, 0, 16)
    with pytest.raises(InvalidArgument):
        sc.linear(ab, m, V, ga, out, swiglu=swiglu, n_offset=8 if flaw == "window" else 0, ldo=cols)
    sc.linear(None, m, W, ga, out, flags=L.LINEAR_A_PREQUANTIZED, swiglu=swiglu)
    be.submit(30000)
    assert np.array_equal(be.read_buffer(out, np.uint16), be.read_buffer(ref, np.uint16))
    W.free(be)
    for buf in (ab, other, out, ref):
        be.free(buf)


def test_output_over_the_activations(backend):
    import thinfer_b200 as T

    be, m, n = backend, 16, 3072
    a, (wc, ws, gw), b = _problem(m, n, n, 9)
    ga = O.global_scale(O.amax_bf16(a))
    W = T.Nvfp4Weight.from_packed(be, wc, ws, gw, b)
    ab, out = be.upload(a), be.allocate(m * n * 2)
    be.scope().linear(ab, m, W, ga, out)
    be.scope().linear(ab, m, W, ga, ab)
    be.submit(30000)
    got, want = (O.bf16_to_f32(be.read_buffer(x, np.uint16)) for x in (ab, out))
    assert rel_fro(got, want) <= 1e-3
    W.free(be)
    be.free(ab)
    be.free(out)
