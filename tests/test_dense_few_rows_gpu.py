"""The dense arm with few rows (the 1-CTA kernel) gives the bits of the CTA-pair kernel, which takes the same rows within a longer operand:
boxes of 32, 64 and 128 rows, tiles of 32, 64 and 128 columns, K that ends within a box or a stage, every epilogue. Up to 16 rows
clusters share K where that pays, and the order of the f32 sums is another one: few results are another bf16 value (2^-8 of them at most)."""
import numpy as np
import pytest

import oracle as O
from conftest import dev_scales_to_canonical, rel_fro
from test_rules import rules  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(256, 32), (1040, 1120), (4736, 96), (4800, 160), (9536, 608), (320, 8992), (2400, 3104), (3008, 4000), (19008, 128)])
@pytest.mark.parametrize("form", ["plain", "gelu", "gate", "swiglu", "quantised"])
def test_few_rows_as_in_a_long_operand(backend, rules, n, k, form):  # noqa: F811
    import torch
    import thinfer_b200 as T
    from thinfer_b200.backend import device_scales_bytes

    be, rng = backend, np.random.default_rng(n + k)
    if form == "quantised":
        n = n // 64 * 64
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    MANY = max(1200, 128 * (sms // -(-n // 128) + 1))  # rows of the long operand: more than a wave of the 1-CTA kernel's tiles
    assert rules.dense_tile(MANY, n, form == "quantised", sms) == 0 and (rules.dense_tile(128, n, form == "quantised", sms) != 0) == (n <= 128 * sms)
    w, b = rng.standard_normal((n, k), np.float32) * np.float32(0.02), O.f32_to_bf16(rng.standard_normal(n, np.float32))
    wc, ws, gw = O.quantize_weight(w)
    W = T.Nvfp4Weight.from_packed(be, wc, ws, gw, b)
    W.prepare_dense(be)
    a = O.f32_to_bf16(rng.standard_normal((MANY, k), np.float32))
    cols = n // 2 if form == "swiglu" else n
    ab, out = be.upload(a), be.allocate((MANY + 1) * cols * 2)
    codes, scales = be.allocate(MANY * n // 2), be.allocate(device_scales_bytes(MANY, n))
    gate, res = be.upload(O.f32_to_bf16(rng.standard_normal(n, np.float32))), be.upload(O.f32_to_bf16(rng.standard_normal((MANY, n), np.float32)))
    kw = dict(act=int(form in ("gelu", "quantised")), swiglu=form == "swiglu", dense_act=True)
    if form == "gate":
        kw.update(gate=gate, residual=res)
    if form == "quantised":
        kw.update(out_nvfp4=(codes, scales, 0.01))
    sc, ref = be.scope(), None
    for m in (MANY, 128, 100, 65, 64, 33, 32, 17, 16, 5, 1):
        be.write_buffer(out, np.full((MANY + 1) * cols, 0x7FC0, np.uint16))
        be.write_buffer(codes, np.full(codes.len, 0xA5, np.uint8))
        be.write_buffer(scales, np.full(scales.len, 0xA5, np.uint8))
        sc.linear(ab, m, W, 0.0, out, **kw)
        be.submit(30000)
        got = be.read_buffer(out, np.uint16).reshape(MANY + 1, cols)
        assert (got[m] == 0x7FC0).all()
        q = be.read_buffer(codes, np.uint8, m * n // 2).reshape(m, n // 2) if form == "quantised" else got[:m]
        s = dev_scales_to_canonical(be.read_buffer(scales, np.uint8, device_scales_bytes(m, n)), m, n) if form == "quantised" else got[:m]
        if ref is None:
            ref, refq, refs = got, q, s
            if form == "plain":
                assert rel_fro(O.bf16_to_f32(got[:16]), O.bf16_to_f32(O.linear(a[:16], 1.0, wc, ws, gw, bias=b, quantize_a=False))) <= 1e-3
        if m > 16:
            assert np.array_equal(got[:m], ref[:m]) and np.array_equal(q, refq[:m]) and np.array_equal(s, refs[:m])
        else:
            for i in range(m):
                assert rel_fro(O.bf16_to_f32(got[i]), O.bf16_to_f32(ref[i])) <= 1e-3
            # another bf16 value is another code at most, and another scale where it is its block's largest: with it all of the block's codes
            assert (q != refq[:m]).mean() <= 0.01 and (s != refs[:m]).mean() <= 0.01
    W.free(be)
    for buf in (ab, out, codes, scales, gate, res):
        be.free(buf)
