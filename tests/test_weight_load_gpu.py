"""Loading a dense weight in one call: the same bytes as upload + quantise + scale layout, from several threads and with a budget, what it
leaves allocated; and pageable writes around the sizes where the staged copy changes its chunks."""
import ctypes as C
import threading

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def _weight(n, k, bf16, seed):
    w = np.random.default_rng(seed).standard_normal((n, k), np.float32) * np.float32(0.02)
    return O.f32_to_bf16(w) if bf16 else w


def _check(be, W, w, bias):
    import thinfer_b200 as T

    V = T.Nvfp4Weight.from_dense(be, w, bias, keep_canonical=True)  # upload, quantise, scale layout: a call each
    assert W.global_scale == V.global_scale
    assert np.array_equal(be.read_buffer(W.codes), be.read_buffer(V.codes))
    assert np.array_equal(be.read_buffer(W.scales_device), be.read_buffer(V.scales_device))
    if bias is None:
        assert W.bias is None
    else:
        assert np.array_equal(be.read_buffer(W.bias, np.uint16), bias)
    V.free(be)


@pytest.mark.parametrize("n,k,bf16", [(2, 32, True), (130, 96, False), (1000, 2080, True), (4104, 3072, True), (12288, 3072, False)])
@pytest.mark.parametrize("budget", [0, 1 << 30])
def test_load_equals_its_parts(n, k, bf16, budget):
    import thinfer_b200 as T

    with T.Backend(0, budget) as be:
        w, bias = _weight(n, k, bf16, n + k), O.f32_to_bf16(np.random.default_rng(n).standard_normal(n, np.float32))
        for b in (bias, None):
            W = T.Nvfp4Weight.from_dense(be, w, b)
            _check(be, W, w, b)
            W.free(be)
        live = be.mem_snapshot()
        assert live["live_weights"] == 0
        assert not budget or live["live_staging"] == 0  # nothing stays where memory is planned


def test_loads_hold_what_they_account_for(backend):
    """Device memory in use against the snapshot's live bytes: whole weights, then their biases alone, then nothing."""
    import torch
    import thinfer_b200 as T

    be, n, k = backend, 16384, 4096  # codes of 32 MiB, scales of 4
    w, bias = _weight(n, k, True, 1), O.f32_to_bf16(np.random.default_rng(2).standard_normal(n, np.float32))
    T.Nvfp4Weight.from_dense(be, w, bias).free(be)
    be.drain_pool()
    live = lambda: sum(v for x, v in be.mem_snapshot().items() if x in ("live_weights", "live_workspace", "live_staging"))
    free0, live0 = torch.cuda.mem_get_info()[0], live()
    grain = 2 << 20  # the driver's pages: an allocation takes whole ones
    used = lambda: free0 - torch.cuda.mem_get_info()[0]
    W = [T.Nvfp4Weight.from_dense(be, w, bias) for _ in range(4)]
    assert used() <= live() - live0 + 13 * grain  # four times three buffers, and the loads' staging
    for x in W:
        be.free(x.codes)
        be.free(x.scales_device)
    be.drain_pool()
    assert live() - live0 == 4 * 2 * n and used() <= live() - live0 + 4 * grain
    for x in W:
        assert np.array_equal(be.read_buffer(x.bias, np.uint16), bias)
        be.free(x.bias)
    assert live() == live0 and used() <= grain


def test_weights_freed_in_another_order(backend):
    """Two dozen weights of 9 MB: every other one read back after its neighbours went."""
    import thinfer_b200 as T

    be, before = backend, backend.mem_snapshot()["live_weights"]
    w = [_weight(4096, 4096, True, i) for i in range(3)]
    W = [T.Nvfp4Weight.from_dense(be, w[i % 3]) for i in range(24)]
    ref = [be.read_buffer(W[i].codes) for i in range(3)]
    for i in range(0, 24, 2):
        W[i].free(be)
    for i in range(1, 24, 2):
        assert np.array_equal(be.read_buffer(W[i].codes), ref[i % 3])
        W[i].free(be)
    assert be.mem_snapshot()["live_weights"] == before


def test_staging_of_loads_is_given_back(backend):
    import thinfer_b200 as T

    be, w = backend, _weight(1000, 2080, True, 3)
    for _ in range(2):
        W = T.Nvfp4Weight.from_dense(be, w)
        be.drain_pool()
        assert be.mem_snapshot()["live_staging"] == 0
        _check(be, W, w, None)
        W.free(be)


def test_loads_of_several_threads(backend):
    import thinfer_b200 as T

    w, out = [_weight(2048 + 128 * i, 1024, i % 2 == 0, i) for i in range(4)], [None] * 4
    def load(i):
        for _ in range(3):
            if out[i]:
                out[i].free(backend)
            out[i] = T.Nvfp4Weight.from_dense(backend, w[i])
    threads = [threading.Thread(target=load, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for W, x in zip(out, w):
        _check(backend, W, x, None)
        W.free(backend)


def test_exported_weight_stays_where_it_is(backend):
    """The address of a buffer is the caller's for as long as it lives; every buffer can be exported."""
    import thinfer_b200 as T
    from thinfer_b200.backend import _check as check

    w, bias = _weight(1024, 1024, True, 7), O.f32_to_bf16(np.ones(1024, np.float32))
    W = T.Nvfp4Weight.from_dense(backend, w, bias)
    for buf in (W.codes, W.scales_device, W.bias):
        handle, p = C.create_string_buffer(64), backend.device_ptr(buf)
        check(backend.lib.tnf_ipc_export(backend._ctx, buf.id, handle))
        assert backend.device_ptr(buf) == p
    _check(backend, W, w, bias)
    W.free(backend)


def test_first_write_of_a_context_costs_no_more_than_it_carries():
    """A megabyte, first and again: what the first makes for itself is not what 24 MB need (7 ms). The least of eight contexts."""
    import time
    import thinfer_b200 as T

    data, extra, backends = np.zeros(1 << 20, np.uint8), [], [T.Backend(0) for _ in range(8)]
    for be in backends:
        buf, t = be.allocate(data.size), [time.perf_counter()]
        for _ in range(4):
            be.write_buffer(buf, data)
            t.append(time.perf_counter())
        took = np.diff(t)
        extra.append(took[0] - took[1:].min())
    for be in backends:
        be.close()
    assert min(extra) < 1e-3


@pytest.mark.parametrize("nbytes", [(1 << 20) - 4, 1 << 20, (2 << 20) - 4, (2 << 20) + 4, (3 << 20) + 8, 8 << 20, (11 << 20) + 12])
def test_pageable_writes(backend, nbytes):
    data = np.random.default_rng(nbytes).integers(0, 256, nbytes + 3, np.uint8)[3:]  # not aligned
    buf = backend.allocate(nbytes + 64)
    backend.write_buffer(buf, np.full(nbytes + 64, 0xA5, np.uint8))
    backend.write_buffer(buf, data, offset=16)
    got = backend.read_buffer(buf)
    assert np.array_equal(got[16: 16 + nbytes], data)
    assert (got[:16] == 0xA5).all() and (got[16 + nbytes:] == 0xA5).all()
    backend.free(buf)


def test_pageable_writes_of_a_new_context():
    """Few bytes go through a few small slots, the first large write makes the others."""
    import thinfer_b200 as T

    with T.Backend(0) as be:
        for nbytes in (1 << 20, (3 << 20) + 8, (5 << 20) + 12, 24 << 20, (3 << 20) + 8):
            data, buf = np.random.default_rng(nbytes).integers(0, 256, nbytes + 3, np.uint8)[3:], be.allocate(nbytes)
            be.write_buffer(buf, data)
            assert np.array_equal(be.read_buffer(buf), data)
            be.free(buf)
