"""The one-launch per-tensor scale (amax_scale_kernel) and the staged copy of large pageable writes: whole numbers and bytes,
so both are compared bit for bit."""
import threading

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


# one 32-element row; below, at and above one block's 4 x 512 loads of 8 elements; remainders; more than the resident grid
@pytest.mark.parametrize("m,k", [(1, 32), (511, 32), (512, 32), (513, 32), (1, 16416), (3, 16384 + 96), (4736, 2080), (6000, 3072)])
@pytest.mark.parametrize("where", [0, -1, None])
def test_scale_of_the_tensor_itself(backend, m, k, where):
    a = np.full((m, k), -0.5, np.float32)
    a.flat[m * k // 2] = np.nan  # dropped, as by the element-wise maximum
    if where is not None:
        a.flat[where] = -7.0
    ab = O.f32_to_bf16(a)
    want = np.float32(7.0 if where is not None else 0.5) / np.float32(2688.0)
    buf = backend.upload(ab)
    for _ in range(2):  # the words are armed again for the next launch
        c, s, g = backend.scope().act_quant(buf, m, k, 0.0, device_layout=True)
        assert np.float32(g) == want
        backend.free(c)
        backend.free(s)
    backend.free(buf)


def test_scale_of_infinite_and_zero_tensors(backend):
    for value, want in ((np.inf, np.inf), (0.0, 1.0), (np.nan, 1.0)):
        buf = backend.upload(O.f32_to_bf16(np.full((64, 64), value, np.float32)))
        c, s, g = backend.scope().act_quant(buf, 64, 64, 0.0)
        assert g == want
        for x in (c, s, buf):
            backend.free(x)


@pytest.mark.parametrize("nbytes", [(8 << 20) + 4, (24 << 20) - 4, 24 << 20, (24 << 20) + 4, (33 << 20) + 12, 100 << 20])
def test_large_pageable_writes(backend, nbytes):
    data = np.random.default_rng(nbytes).integers(0, 256, nbytes, np.uint8)
    buf = backend.allocate(nbytes + 64)
    backend.write_buffer(buf, np.full(nbytes + 64, 0xA5, np.uint8))
    backend.write_buffer(buf, data, offset=16)
    got = backend.read_buffer(buf)
    assert np.array_equal(got[16: 16 + nbytes], data)
    assert (got[:16] == 0xA5).all() and (got[16 + nbytes:] == 0xA5).all()
    backend.free(buf)


def test_large_writes_from_several_threads(backend):
    """One of them has the pinned slots, the others copy the plain way."""
    datas = [np.random.default_rng(i).integers(0, 256, (26 << 20) + 4 * i, np.uint8) for i in range(4)]
    bufs = [backend.allocate(d.nbytes) for d in datas]
    threads = [threading.Thread(target=backend.write_buffer, args=(b, d)) for b, d in zip(bufs, datas)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for b, d in zip(bufs, datas):
        assert np.array_equal(backend.read_buffer(b), d)
        backend.free(b)


@pytest.mark.parametrize("n_threads", [8, 72])  # 72: more calls wait for a scale than there are words to report it in
def test_own_scales_of_several_threads(backend, n_threads):
    """Threads that share a context quantise tensors of very different magnitude, each with its own scale: codes, block scales and
    the reported scale belong to the same tensor, in every interleaving of the calls' launches."""
    import ctypes as C

    from thinfer_b200 import _lib as L

    be, m, k = backend, 96, 256
    a = [O.f32_to_bf16(np.random.default_rng(i).standard_normal((m, k)).astype(np.float32) * np.float32(4.0 ** (i % 9 - 4))) for i in range(n_threads)]
    g = [O.global_scale(O.amax_bf16(x)) for x in a]
    bufs = [(be.upload(x), be.allocate(m * k // 2), be.allocate(m * k // 16)) for x in a]
    wrong = []

    def work(i):
        src, codes, scales = bufs[i]
        used = C.c_float()
        for _ in range(300 if n_threads == 8 else 40):
            st = be.lib.tnf_quantize_act(be._ctx, src, m, k, 0.0, L.SCALES_CANONICAL, codes, scales, C.byref(used))
            if st != 0 or used.value != np.float32(g[i]):
                wrong.append((i, st, used.value))
        # without asking for the scale: the launches of the threads run into one another
        for _ in range(50):
            be.lib.tnf_quantize_act(be._ctx, src, m, k, 0.0, L.SCALES_CANONICAL, codes, scales, None)

    for _ in range(6):  # the codes are looked at after each round: the last call of each thread
        threads = [threading.Thread(target=work, args=(i,)) for i in range(n_threads)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        be.submit(30000)
        for i in range(n_threads):
            oc, os_ = O.quantize_act(a[i], g[i])
            assert np.array_equal(be.read_buffer(bufs[i][1]).reshape(m, k // 2), oc), i
            assert np.array_equal(be.read_buffer(bufs[i][2]).reshape(m, k // 16), os_), i
    assert not wrong
    for group in bufs:
        for b in group:
            be.free(b)
