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


@pytest.mark.parametrize("nbytes", [(8 << 20) - 4, 8 << 20, (8 << 20) + 4, (33 << 20) + 12, 100 << 20])
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
    datas = [np.random.default_rng(i).integers(0, 256, (12 << 20) + 4 * i, np.uint8) for i in range(4)]
    bufs = [backend.allocate(d.nbytes) for d in datas]
    threads = [threading.Thread(target=backend.write_buffer, args=(b, d)) for b, d in zip(bufs, datas)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for b, d in zip(bufs, datas):
        assert np.array_equal(backend.read_buffer(b), d)
        backend.free(b)
