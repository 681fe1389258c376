"""Banded tile order of the pair kernel (an A too large for L2): the order changes no bit, so the whole linear equals the same
rows computed in slices that are too small for bands. Row tiles that do not fill the last band, ragged rows and columns, halves
of the last wave's tiles; both rules (a W that stays in L2, and one that does not)."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,dense", [
    (15000, 528, 1024, False),   # 8.6 MB of A: one band and a short one
    (9000, 3072, 4096, False),   # bands of 14 row tiles, 36 in all; 432 tiles: the last wave in halves
    (7000, 1040, 8192, False),   # bands of 7, ragged columns
    (2600, 272, 65536, False),   # a row tile as large as a band: bands of one
    (14100, 4400, 4096, True),   # bf16 activations, a W of 36 MB: bands of 54 MB
])
def test_bands_change_no_bit(backend, m, n, k, dense):
    import thinfer_b200 as T
    from thinfer_b200 import _lib as L

    be = backend
    rng = np.random.default_rng(m)
    a = O.f32_to_bf16(rng.standard_normal((m, k), np.float32))
    W = T.Nvfp4Weight.from_dense(be, rng.standard_normal((n, k), np.float32) * np.float32(0.02), O.f32_to_bf16(rng.standard_normal(n, np.float32)))
    if dense:
        W.prepare_dense(be)
    ab, out, part = be.upload(a), be.allocate(m * n * 2), be.allocate(m * n * 2)
    sc, g = be.scope(), 0.002
    sc.linear(ab, m, W, g, out, dense_act=dense)
    step = 1024 if k < 65536 else 256  # too few tiles for the pair kernel's bands, some of them on the 1-CTA kernel
    for r in range(0, m, step):
        rows = min(step, m - r)
        sc.linear(L.Buf(ab.id, r * k * 2, rows * k * 2), rows, W, g, L.Buf(part.id, r * n * 2, rows * n * 2), dense_act=dense)
    be.submit(60000)
    got, want = be.read_buffer(out, np.uint16), be.read_buffer(part, np.uint16)
    assert np.array_equal(got, want)
    W.free(be)
    for buf in (ab, out, part):
        be.free(buf)
