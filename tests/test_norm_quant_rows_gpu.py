"""The warp-per-row form of tnf_norm_modulate_quantize (about ten rows per SM and more, up to 3072 columns; the shape (2369, 2048)
is just past it, in a second round of rows that is nearly empty), on the checks of test_norm_quant_gpu.py: the bf16 result against the CPU restatement (row sums in another order), the NVFP4 copy bit for bit
against the oracle quantiser on the kernel's own bf16 output."""
import numpy as np
import pytest

import oracle as O
from conftest import dev_scales_to_canonical, rel_fro
from test_norm_quant_gpu import G_OUT, _inputs, _run

pytestmark = pytest.mark.gpu


# one block per row; a lane short of a warp, a warp, one more; every count of blocks per lane; 1, 2 and 3 rows per warp
@pytest.mark.parametrize("m,k", [(1480, 16), (1481, 496), (1500, 512), (1487, 528), (1600, 1040), (2369, 2048), (2400, 2064),
                                 (1999, 2576), (4737, 3056), (4352, 3072), (1554, 3072), (2724, 2048), (2800, 2064)])
@pytest.mark.parametrize("mod", [True, False])
def test_warp_per_row(backend, m, k, mod):
    x, s, t = _inputs(m, k, m + k)
    if not mod:
        s = t = None
    y, c, dev = _run(backend, x, s, t, False)
    want = O.norm_modulate(x, s, t, 1e-6, 1.0, chain=False) if mod else O.ref_layernorm(x, 1e-6)
    assert not np.isnan(O.bf16_to_f32(y)).any()
    assert rel_fro(O.bf16_to_f32(y), O.bf16_to_f32(want)) <= 1e-3
    assert (y == want).mean() >= 0.98
    oc, os_ = O.quantize_act(y, G_OUT)
    assert np.array_equal(c, oc)
    assert np.array_equal(dev_scales_to_canonical(dev, m, k), os_)
    assert np.array_equal(dev, O.scales_to_device_layout(os_))  # padding bytes are zero
    _, c2, dev2 = _run(backend, x, s, t, False, want_bf16=False)
    assert np.array_equal(c, c2) and np.array_equal(dev, dev2)
