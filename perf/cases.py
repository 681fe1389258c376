"""The workloads this library is timed on, through its public Python surface.

Sizes are those of the repository's own benchmark and tests (Qwen-Image-shaped block linears at 4352 tokens, Wan-5B-shaped
FFN at 6630 and 26520 tokens, the M = 1 modulation linear, the 256 x 3072 x 3072 linear) and generic ragged ones between
them. Weights are N(0, 0.02), activations N(0, 1), biases N(0, 0.01), made from a seed on the device.

    listed()              the named cases
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs, weights and output buffers
    run(state)            one pass; returns the outputs as torch views of the library's buffers
    work(case)            bytes and floating-point operations one pass cannot do without
    exact(case, seed)     the outputs in float64, without the library's code
    tolerance(case)       how far another correct implementation of the same precision may be off
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import thinfer_b200 as T
from thinfer_b200 import _lib as L
from thinfer_b200.backend import _check, device_scales_bytes
from thinfer_b200.residency import LayerStack, StackLinearSpec

HEAD = 128


# ---- cases ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # AdaLN modulation of one timestep: the smallest call of a DiT block, one row against a wide weight
        dict(name="modulation_m1", kind="linear", m=1, n=18432, k=3072, act=0, gate=False, dense=False, swiglu=False),
        # a lone small linear (text-side or refiner projection): latency and launches count
        dict(name="linear_256", kind="linear", m=256, n=3072, k=3072, act=0, gate=False, dense=False, swiglu=False),
        # gated FFN-up of a text encoder or refiner block at a ragged token count, SwiGLU fused
        dict(name="swiglu_1111", kind="linear", m=1111, n=16384, k=3072, act=0, gate=False, dense=False, swiglu=True),
        # MLP-down of a site that keeps its activations in bf16 (dense arm)
        dict(name="dense_down_4352", kind="linear", m=4352, n=3072, k=12288, act=0, gate=False, dense=True, swiglu=False),
        # one whole image-transformer block at 1024 x 1024: norm + modulate + quantise, four linears, attention, gated residuals
        dict(name="block_4352", kind="block", m=4352, hidden=3072, ffn=12288),
        # video FFN at a ragged token count: quantise, up + GELU emitting NVFP4, down
        dict(name="ffn_6630", kind="ffn", m=6630, k=3072, ffn=14336),
        # the same FFN over a batch of four clips: the largest contraction
        dict(name="ffn_26520", kind="ffn", m=26520, k=3072, ffn=14336),
        # joint attention over a long sequence
        dict(name="sdpa_16384", kind="sdpa", b=1, s_q=16384, s_k=16384, heads=12, kv_heads=12),
        # cross attention of video tokens to a short text sequence
        dict(name="sdpa_cross_6630x512", kind="sdpa", b=1, s_q=6630, s_k=512, heads=24, kv_heads=24),
        # bringing a bf16 checkpoint tensor in: upload, quantise, device scale layout
        dict(name="load_weight_12288", kind="load", n=12288, k=3072, bf16=True),
        # activation quantiser with a scale taken from the tensor itself (calibration, uncalibrated sites)
        dict(name="quantise_dynamic_4352", kind="quantise", m=4352, k=3072, device_layout=True),
        # layer stack streamed from pinned host memory under a weight budget of about half its size
        dict(name="stack_streamed", kind="stack", layers=8, m=4352, hidden=3072, ffn=12288, resident=0.53),
    ]


def _log_int(rng, lo, hi, step=1):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step
    return max(step, min(hi // step * step, max(lo, v)))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "linear", "block", "ffn", "ffn", "sdpa", "sdpa", "load", "quantise", "stack"])
    if kind == "linear":
        arm = rng.choice(["plain", "plain", "plain", "gelu", "gate", "dense", "swiglu"])
        m, n, k = _log_int(rng, 1, 8192), _log_int(rng, 256, 18432, 16), _log_int(rng, 256, 14336, 32)
        return dict(kind=kind, m=m, n=n, k=k, act=int(arm == "gelu"), gate=arm == "gate", dense=arm == "dense", swiglu=arm == "swiglu")
    if kind == "block":
        hidden = 128 * rng.randint(8, 24)
        return dict(kind=kind, m=_log_int(rng, 256, 4352), hidden=hidden, ffn=4 * hidden)
    if kind == "ffn":
        return dict(kind=kind, m=_log_int(rng, 64, 26520), k=_log_int(rng, 1024, 3072, 64), ffn=_log_int(rng, 2048, 14336, 64))
    if kind == "sdpa":
        s_q, s_k, heads = _log_int(rng, 128, 16384), _log_int(rng, 32, 16384), rng.randint(1, 12)
        group = rng.choice([1, 1, 2])
        return dict(kind=kind, b=rng.choice([1, 1, 2]) if s_q * s_k < (1 << 26) else 1, s_q=s_q, s_k=s_k, heads=heads * group, kv_heads=heads)
    if kind == "load":
        return dict(kind=kind, n=_log_int(rng, 512, 12288, 8), k=_log_int(rng, 512, 3072, 32), bf16=rng.random() < 0.7)
    if kind == "quantise":
        return dict(kind=kind, m=_log_int(rng, 16, 8192), k=_log_int(rng, 256, 12288, 32), device_layout=rng.random() < 0.7)
    hidden = 128 * rng.randint(8, 24)
    return dict(kind="stack", layers=rng.randint(4, 8), m=_log_int(rng, 256, 4352), hidden=hidden, ffn=4 * hidden, resident=round(rng.uniform(0.55, 0.9), 2))


# ---- device buffers --------------------------------------------------------------------------------------------------
_backend = None


def _be() -> T.Backend:
    """One backend per process, as a program that serves a model keeps it."""
    global _backend
    if _backend is None:
        _backend = T.Backend(0)
    return _backend


class _Mem:
    """A library buffer that is given back with its last user; torch views hold it through __cuda_array_interface__."""

    def __init__(self, nbytes, category=L.CAT_WORKSPACE, buf=None):
        self.buf = buf if buf is not None else _be().allocate_in(max(int(nbytes), 256), category)
        self.nbytes = int(nbytes)
        self.ptr = _be().device_ptr(self.buf)

    @property
    def __cuda_array_interface__(self):
        return {"shape": (self.nbytes,), "typestr": "|u1", "data": (self.ptr, False), "version": 2}

    def view(self, dtype, *shape):
        return torch.as_tensor(self, device="cuda:0").view(dtype).view(*shape)

    def __del__(self):
        try:
            _be().free(self.buf)
        except Exception:
            pass


class _State:
    def __init__(self, case, seed):
        self.case, self.be = case, _be()
        self.scope = self.be.scope()
        self.gen = torch.Generator(device="cuda:0")
        self.gen.manual_seed(int(seed))
        self.mem = {}

    def randn(self, *shape):
        return torch.randn(*shape, device="cuda:0", generator=self.gen)

    def new(self, name, nbytes, category=L.CAT_WORKSPACE):
        self.mem[name] = _Mem(nbytes, category)
        return self.mem[name].buf

    def tensor(self, name, values):
        """A bf16 input buffer filled with `values`."""
        buf = self.new(name, values.numel() * 2)
        self.mem[name].view(torch.bfloat16, *values.shape).copy_(values.to(torch.bfloat16))
        return buf

    def out(self, name, rows, cols):
        """A bf16 output buffer and its torch view."""
        buf = self.new(name, rows * cols * 2)
        return buf, self.mem[name].view(torch.bfloat16, rows, cols)

    def weight(self, name, n, k, dense=False):
        be, src = self.be, _Mem(n * k * 2, L.CAT_STAGING)
        src.view(torch.bfloat16, n, k).copy_((self.randn(n, k) * 0.02).to(torch.bfloat16))
        codes, scales = self.new(name + ".codes", n * k // 2, L.CAT_WEIGHTS), self.new(name + ".scales", device_scales_bytes(n, k), L.CAT_WEIGHTS)
        canonical, g = _Mem(n * k // 16, L.CAT_STAGING), C.c_float()
        torch.cuda.synchronize()
        _check(be.lib.tnf_quantize_weight(be._ctx, src.buf, L.DTYPE_BF16, n, k, codes, canonical.buf, C.byref(g)))
        _check(be.lib.tnf_prepare_scales(be._ctx, canonical.buf, n, k, scales))
        w = T.Nvfp4Weight(n, k, codes, scales, float(g.value), self.tensor(name + ".bias", self.randn(n) * 0.01), None)
        if dense:
            self.mem[name + ".dense"] = _Mem(0, buf=w.prepare_dense(be))
        be.submit()
        return w


def _scale_of(amax):
    """Per-tensor scale of a calibrated activation whose largest magnitude is `amax`."""
    return float(amax) / (6.0 * 448.0)


# ---- prepare / run -----------------------------------------------------------------------------------------------------
def prepare(case, seed):
    st = _State(case, seed)
    globals()["_prepare_" + case["kind"]](st, case)
    torch.cuda.synchronize()
    return st


def run(st):
    return st.call()


def _prepare_linear(st, c):
    m, n, k = c["m"], c["n"], c["k"]
    w = st.weight("w", n, k, dense=c["dense"])
    x = st.randn(m, k)
    g = _scale_of(x.abs().max())
    a = st.tensor("a", x)
    cols = n // 2 if c["swiglu"] else n
    out, view = st.out("out", m, cols)
    gate = residual = None
    if c["gate"]:
        gate, residual = st.tensor("gate", st.randn(n) * 0.5), st.tensor("residual", st.randn(m, n))

    def call():
        st.scope.linear(a, m, w, g, out, act=c["act"], gate=gate, residual=residual, dense_act=c["dense"], swiglu=c["swiglu"])
        return view

    st.call = call


def _prepare_ffn(st, c):
    m, k, ffn = c["m"], c["k"], c["ffn"]
    up, down = st.weight("up", ffn, k), st.weight("down", k, ffn)
    x = st.randn(m, k)
    g_x, g_h = _scale_of(x.abs().max()), _scale_of(5.5 * 0.02 * math.sqrt(k))
    a = st.tensor("x", x)
    h = (st.new("h.codes", m * ffn // 2), st.new("h.scales", device_scales_bytes(m, ffn)), g_h)
    y, view = st.out("y", m, k)

    def call():
        st.scope.linear(a, m, up, g_x, None, act=L.ACT_GELU_TANH, out_nvfp4=h)
        st.scope.matmul(h[0], h[1], m, down, g_h, y)
        return view

    st.call = call


def _prepare_block(st, c):
    m, d, ffn = c["m"], c["hidden"], c["ffn"]
    heads, sc = d // HEAD, st.scope
    w_qkv, w_out, w_up, w_down = (st.weight(nm, n, k) for nm, n, k in (("w_qkv", 3 * d, d), ("w_out", d, d), ("w_up", ffn, d), ("w_down", d, ffn)))
    x = st.tensor("x", st.randn(m, d))
    mod = [[st.tensor(f"{nm}{i}", st.randn(d) * s) for nm, s in (("shift", 0.2), ("scale", 0.3), ("gate", 0.1))] for i in (0, 1)]
    xc, xs = st.new("x.codes", m * d // 2), st.new("x.scales", device_scales_bytes(m, d))
    ac, as_ = st.new("attn.codes", m * d // 2), st.new("attn.scales", device_scales_bytes(m, d))
    uc, us = st.new("up.codes", m * ffn // 2), st.new("up.scales", device_scales_bytes(m, ffn))
    qkv = st.new("qkv", m * 3 * d * 2)
    win = [L.Buf(qkv.id, i * d * 2, m * 3 * d * 2 - i * d * 2) for i in range(3)]
    (h1, v1), (y, v2) = st.out("h1", m, d), st.out("y", m, d)
    s_lin = 0.02 * math.sqrt(d)  # spread of a linear's output for inputs of spread 1
    g_x, g_up = _scale_of(7.0), _scale_of(5.5 * s_lin)
    # the attention output averages v over the rows: what is left is the part of v the shift gives every row, and noise
    g_at = _scale_of(5.5 * s_lin * math.sqrt(0.2 ** 2 + min(1.0, math.exp(min(s_lin ** 4, 3.0)) / m)))

    def call():
        sc.norm_modulate_quant(x, m, d, g_x, xc, xs, scale=mod[0][1], shift=mod[0][0])
        sc.matmul(xc, xs, m, w_qkv, g_x, qkv)
        sc.sdpa(win[0], win[1], win[2], None, 1, m, m, heads, heads, HEAD ** -0.5, out_nvfp4=(ac, as_, g_at), q_ld=3 * d, kv_ld=3 * d)
        sc.matmul(ac, as_, m, w_out, g_at, h1, gate=mod[0][2], residual=x)
        sc.norm_modulate_quant(h1, m, d, g_x, xc, xs, scale=mod[1][1], shift=mod[1][0])
        sc.matmul(xc, xs, m, w_up, g_x, None, act=L.ACT_GELU_TANH, out_nvfp4=(uc, us, g_up))
        sc.matmul(uc, us, m, w_down, g_up, y, gate=mod[1][2], residual=h1)
        return v1, v2

    st.call = call


def _prepare_sdpa(st, c):
    b, s_q, s_k, hq, hk = c["b"], c["s_q"], c["s_k"], c["heads"], c["kv_heads"]
    q, k, v = (st.tensor(nm, st.randn(b * s, h * HEAD)) for nm, s, h in (("q", s_q, hq), ("k", s_k, hk), ("v", s_k, hk)))
    out, view = st.out("out", b * s_q, hq * HEAD)

    def call():
        st.scope.sdpa(q, k, v, out, b, s_q, s_k, hq, hk, HEAD ** -0.5)
        return view

    st.call = call


def _prepare_load(st, c):
    n, k, be = c["n"], c["k"], st.be
    w = st.randn(n, k) * 0.02
    host = w.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16) if c["bf16"] else w.cpu().numpy()
    bias = (st.randn(n) * 0.01).to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)

    def call():
        w = T.Nvfp4Weight.from_dense(be, host, bias)
        codes, scales, b = _Mem(w.codes.len, buf=w.codes), _Mem(w.scales_device.len, buf=w.scales_device), _Mem(w.bias.len, buf=w.bias)
        return codes.view(torch.uint8, n, k // 2), scales.view(torch.uint8, -1), b.view(torch.bfloat16, n), w.global_scale

    st.call = call


def _prepare_quantise(st, c):
    m, k, be, dev = c["m"], c["k"], st.be, c["device_layout"]
    a = st.tensor("a", st.randn(m, k))
    codes, scales = st.new("codes", m * k // 2), st.new("scales", device_scales_bytes(m, k) if dev else m * k // 16)
    views = st.mem["codes"].view(torch.uint8, m, k // 2), st.mem["scales"].view(torch.uint8, -1)
    layout, g = L.SCALES_DEVICE if dev else L.SCALES_CANONICAL, C.c_float()

    def call():
        _check(be.lib.tnf_quantize_act(be._ctx, a, m, k, 0.0, layout, codes, scales, C.byref(g)))
        return views[0], views[1], float(g.value)

    st.call = call


class _Stack:
    """A LayerStack that goes with its last user."""

    def __init__(self, *args):
        self.stack = LayerStack(*args)

    def __del__(self):
        try:
            self.stack.close()
        except Exception:
            pass


def _prepare_stack(st, c):
    d, ffn, m, be = c["hidden"], c["ffn"], c["m"], st.be
    specs = [StackLinearSpec(3 * d, d, 0, True, 0, 0), StackLinearSpec(d, d, 0, True, 2, 0),
             StackLinearSpec(ffn, d, L.ACT_GELU_TANH, True, 1, 0), StackLinearSpec(d, ffn, 0, True, 1, 0)]
    holder = _Stack(be, c["layers"], specs, [m], d)
    stack = holder.stack
    for layer in range(c["layers"]):
        for j, s in enumerate(specs):
            w = st.weight("w", s.n, s.k)
            stack.pack(layer, j, be.read_buffer(w.codes), be.read_buffer(w.scales_device), w.global_scale, be.read_buffer(w.bias, np.uint16, s.n))
    stack.build(weight_budget=int(c["resident"] * stack.layer_bytes * c["layers"]), ring_slots=2)
    x, aux = st.tensor("x", st.randn(m, d)), st.tensor("aux", st.randn(m, d))
    out, view = st.out("out", m, d)
    st.holder = holder

    def call():
        stack.step([x], [out], _scale_of(5.5), aux=[aux])
        return view

    st.call = call


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------
def _q(rows, k):
    """Bytes of an NVFP4 operand: codes and block scales."""
    return rows * k * 9 // 16


def _linear_work(m, n, k, w_bytes=None):
    return 2 * m * k + (_q(n, k) if w_bytes is None else w_bytes) + 2 * n + 2 * m * n, 2 * m * n * k


def work(case):
    c = case
    if c["kind"] == "linear":
        b, f = _linear_work(c["m"], c["n"], c["k"], 2 * c["n"] * c["k"] if c["dense"] else None)
        if c["swiglu"]:
            b -= c["m"] * c["n"]
        if c["gate"]:
            b += 2 * c["m"] * c["n"] + 2 * c["n"]
    elif c["kind"] == "ffn":
        m, k, n = c["m"], c["k"], c["ffn"]
        b, f = 4 * m * k + 2 * _q(n, k) + 2 * (n + k), 4 * m * n * k
    elif c["kind"] == "block":
        m, d, n = c["m"], c["hidden"], c["ffn"]
        b, f = 2 * m * d * 3 + _q(4 * d, d) + 2 * _q(n, d), 2 * m * d * (4 * d + 2 * n) + 4 * m * m * d
    elif c["kind"] == "sdpa":
        b = 2 * HEAD * c["b"] * (2 * c["s_q"] * c["heads"] + 2 * c["s_k"] * c["kv_heads"])
        f = 4 * c["b"] * c["heads"] * c["s_q"] * c["s_k"] * HEAD
    elif c["kind"] == "load":
        b, f = c["n"] * c["k"] * (2 if c["bf16"] else 4) + _q(c["n"], c["k"]), 0
    elif c["kind"] == "quantise":
        b, f = 2 * c["m"] * c["k"] + _q(c["m"], c["k"]), 0
    else:
        m, d, n = c["m"], c["hidden"], c["ffn"]
        b, f = c["layers"] * (_q(4 * d, d) + 2 * _q(n, d)) + 6 * m * d, c["layers"] * 2 * m * d * (4 * d + 2 * n)
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits, without the library ------------------------------------------------------------------------
_E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0]


def _bf16(x):
    return x.to(torch.bfloat16).double()


def _nvfp4(x, g):
    """What the NVFP4 copy of a bf16 matrix stands for, without the per-tensor scale g: code times block scale, in float64.
    The format's own operations are 32-bit ones: scale = e4m3(max * (1 / (6 g))), code = e2m1(x * (1 / (scale * g)))."""
    one, out = torch.ones((), device=x.device), torch.empty(x.shape, dtype=torch.float64, device=x.device)
    g = one * g
    mid = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=x.device)
    values = torch.tensor(_E2M1, dtype=torch.float64, device=x.device)
    for i in range(0, x.shape[0], 2048):
        b = x[i:i + 2048].float().reshape(-1, 16)
        s = (b.abs().amax(1, keepdim=True) * (one / (6.0 * g))).clamp(max=448.0).to(torch.float8_e4m3fn).float()
        y = b * torch.where(s > 0, one / (s * g), 0.0)
        a = y.abs()
        code = torch.bucketize(a, mid)  # a tie stays in the lower interval ...
        for t in (1, 3, 5):  # ... and goes up where the lower code is odd
            code = torch.where(a == mid[t], t + 1, code)
        out[i:i + 2048] = (torch.copysign(values[code], y.double()) * s.double()).reshape(-1, x.shape[1])
    return out


def _gelu64(v):
    return 0.5 * v * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (v + 0.044715 * v ** 3)))


class _Draws:
    """The numbers prepare() draws, in its order."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda:0")
        self.gen.manual_seed(int(seed))

    randn = _State.randn

    def tensor(self, values):
        return values.to(torch.bfloat16).double()

    def weight(self, n, k):
        """(code times block scale, per-tensor scale, bias)"""
        w = (self.randn(n, k) * 0.02).to(torch.bfloat16)
        g = float(np.float32(float(w.float().abs().max())) / np.float32(2688.0))  # a true f32 division: one unit in the last place decides ties
        return _nvfp4(w, g), g, self.tensor(self.randn(n) * 0.01)


def _linear64(a, g_a, w, act=0):
    v = (a @ w[0].T) * (g_a * w[1]) + w[2]
    return _gelu64(v) if act else v


def _attention64(q, k, v, heads, kv_heads):
    out = torch.empty_like(q)
    for h in range(heads):
        j = h * kv_heads // heads
        cols, kv = slice(h * HEAD, (h + 1) * HEAD), slice(j * HEAD, (j + 1) * HEAD)
        for i in range(0, q.shape[0], 4096):
            s = q[i:i + 4096, cols] @ k[:, kv].T * HEAD ** -0.5
            out[i:i + 4096, cols] = torch.softmax(s, 1) @ v[:, kv]
    return out


def _f32(g):
    return float(np.float32(g))


def exact(case, seed):
    """run()'s outputs in float64; what the path stores in bf16 or NVFP4 between two kernels is rounded to that format."""
    c, d = case, _Draws(seed)
    if c["kind"] == "linear":
        m, n, k = c["m"], c["n"], c["k"]
        w = d.weight(n, k)
        x = d.randn(m, k)
        g = _f32(_scale_of(x.abs().max()))
        v = _linear64(d.tensor(x), 1.0, w, c["act"]) if c["dense"] else _linear64(_nvfp4(x.to(torch.bfloat16), g), g, w, c["act"])
        if c["swiglu"]:
            v = v[:, 0::2] * torch.sigmoid(v[:, 0::2]) * v[:, 1::2]
        if c["gate"]:
            gate = d.tensor(d.randn(n) * 0.5)
            v = d.tensor(d.randn(m, n)) + gate * v
        return v
    if c["kind"] == "ffn":
        m, k, ffn = c["m"], c["k"], c["ffn"]
        up, down = d.weight(ffn, k), d.weight(k, ffn)
        x = d.randn(m, k)
        g_x, g_h = _f32(_scale_of(x.abs().max())), _f32(_scale_of(5.5 * 0.02 * math.sqrt(k)))
        a, out = _nvfp4(x.to(torch.bfloat16), g_x), torch.empty(m, k, dtype=torch.float64, device=x.device)
        for i in range(0, m, 8192):
            h = _linear64(a[i:i + 8192], g_x, up, 1).to(torch.bfloat16)
            out[i:i + 8192] = _linear64(_nvfp4(h, g_h), g_h, down)
        return out
    if c["kind"] == "block":
        m, dim, ffn = c["m"], c["hidden"], c["ffn"]
        w_qkv, w_out, w_up, w_down = (d.weight(n, k) for n, k in ((3 * dim, dim), (dim, dim), (ffn, dim), (dim, ffn)))
        x = d.tensor(d.randn(m, dim))
        mod = [[d.tensor(d.randn(dim) * s) for s in (0.2, 0.3, 0.1)] for _ in (0, 1)]
        s_lin = 0.02 * math.sqrt(dim)
        g_x, g_up = _f32(_scale_of(7.0)), _f32(_scale_of(5.5 * s_lin))
        g_at = _f32(_scale_of(5.5 * s_lin * math.sqrt(0.2 ** 2 + min(1.0, math.exp(min(s_lin ** 4, 3.0)) / m))))

        def normed(v, shift, scale):
            n = (v - v.mean(1, keepdim=True)) / torch.sqrt(v.var(1, unbiased=False, keepdim=True) + 1e-6)
            return _nvfp4((n * (1.0 + scale) + shift).to(torch.bfloat16), g_x)

        qkv = _bf16(_linear64(normed(x, mod[0][0], mod[0][1]), g_x, w_qkv))
        at = _attention64(qkv[:, :dim], qkv[:, dim:2 * dim], qkv[:, 2 * dim:], dim // HEAD, dim // HEAD)
        h1 = x + mod[0][2] * _linear64(_nvfp4(at.to(torch.bfloat16), g_at), g_at, w_out)
        up = _linear64(normed(_bf16(h1), mod[1][0], mod[1][1]), g_x, w_up, 1)
        return h1, _bf16(h1) + mod[1][2] * _linear64(_nvfp4(up.to(torch.bfloat16), g_up), g_up, w_down)
    if c["kind"] == "sdpa":
        b, s_q, s_k, hq, hk = c["b"], c["s_q"], c["s_k"], c["heads"], c["kv_heads"]
        q, k, v = (d.tensor(d.randn(b * s, h * HEAD)) for s, h in ((s_q, hq), (s_k, hk), (s_k, hk)))
        return torch.cat([_attention64(q[i * s_q:(i + 1) * s_q], k[i * s_k:(i + 1) * s_k], v[i * s_k:(i + 1) * s_k], hq, hk) for i in range(b)])
    if c["kind"] == "stack":
        dim, ffn, m = c["hidden"], c["ffn"], c["m"]
        shapes = ((3 * dim, dim), (dim, dim), (ffn, dim), (dim, ffn))
        for _ in range(c["layers"]):  # only the last layer's weights reach the result: every layer starts from the auxiliary input
            w = [d.weight(n, k) for n, k in shapes]
        d.randn(m, dim)
        g, v = _f32(_scale_of(5.5)), d.randn(m, dim)
        for wj, act in zip(w[1:], (0, 1, 0)):
            v = _linear64(_nvfp4(v.to(torch.bfloat16), g), g, wj, act)
        return v
    return None  # codes, scales and bytes: the same everywhere


# Measured against a float64 evaluation of the same contract (dequantised operands, exact softmax, tanh and GELU; every tensor
# that the path rounds to bf16 or NVFP4 rounded there too): relative 2-norm error and largest error over the root mean square.
# Stated at about four times that. A linear alone is the order of its f32 sums, then one bf16 rounding; attention adds its bf16
# probabilities; where a result is quantised to FP4 for the next linear, a last-bit difference flips a code now and then.
_TOLERANCE = {
    "linear": {"rel": 6e-4, "max": 0.03},  # 1.4e-4 (dense, K = 12288), 8.7e-5 (tanh approximation), 0.9e-5 (FP4); 0.008
    "ffn": {"rel": 4e-3, "max": 0.15},     # 1.0e-3; 0.037
    "sdpa": {"rel": 0.01, "max": 0.07},    # 2.5e-3; 0.017
    "block": {"rel": 0.03, "max": 0.55},    # 7.6e-3 (four FP4 hand-overs behind the attention, gated residuals); 0.14
    "stack": {"rel": 5e-3, "max": 0.6},    # 1.1e-3; 0.14
}


def tolerance(case):
    return _TOLERANCE.get(case["kind"], "exact")  # a quantiser's codes, scales and per-tensor scale are exact
