"""The 1-CTA GEMM's boxes of 32, 64 and 128 rows of A: what shared memory holds behind the box, from the launch before, must not show."""
import numpy as np
import pytest

import oracle as O
from conftest import rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(4104, 3072), (304, 2272), (5120, 8992)])
@pytest.mark.parametrize("swiglu", [False, True])
def test_rows_around_a_box(backend, n, k, swiglu):
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    be, rng, g = backend, np.random.default_rng(n + k), 0.002
    n = n // 16 * 16
    w = rng.standard_normal((n, k), np.float32) * np.float32(0.02)
    W = T.Nvfp4Weight.from_dense(be, w)
    a = O.f32_to_bf16(rng.standard_normal((129, k), np.float32))
    cols = n // 2 if swiglu else n
    ab, out = be.upload(a), be.allocate(129 * cols * 2)
    sc, flags = be.scope(), L.LINEAR_A_PREQUANTIZED  # the skinny kernels, up to 16 rows, have bits of their own
    ref = None
    for m in (128, 129, 127, 65, 64, 63, 33, 32, 31, 17, 1, 64, 128):
        sc.act_quant_shared(ab, m, k, g)
        sc.linear(None, m, W, g, out, flags=flags, swiglu=swiglu)
        be.submit(30000)
        got = be.read_buffer(out, np.uint16, m * cols).reshape(m, cols)
        if ref is None:
            ref = got
            wc, ws, gw = O.quantize_weight(w)
            want = O.bf16_to_f32(O.linear(a[:128], g, wc, ws, gw))
            if swiglu:
                x, y = want[:, 0::2].astype(np.float64), want[:, 1::2]
                want = x / (1.0 + np.exp(-x)) * y
            assert rel_fro(O.bf16_to_f32(got), want) <= (8e-3 if swiglu else 1e-3)  # SwiGLU here of bf16-rounded halves: two roundings of 2^-9
        assert np.array_equal(got[:128], ref[:m])
    W.free(be)
    be.free(ab)
    be.free(out)
