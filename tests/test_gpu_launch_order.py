"""Kernels that start before their predecessor on the stream has ended: what they read and how long they wait."""
import pytest
import torch

from convnn_b200 import _capi, ops
from gpu_util import DEV

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def rnd(*shape, seed, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV) * scale).to(BF)


def spec_of(T, D, H=1, K=9):
    return ops.LayerSpec(D, H, K, "all", "cosine", "depthwise", True, False, T)


def _mlp(M, D=192, DM=768):
    x, w1 = rnd(M, D, seed=1), rnd(DM, D, seed=2, scale=D ** -0.5)
    wf, wx = ops.fold_layernorm(w1, rnd(DM, seed=3), rnd(D, seed=4), rnd(D, seed=5))
    return x, ops.row_moments(x), wf, wx, rnd(D, DM, seed=6, scale=DM ** -0.5), rnd(D, seed=7)


def _similarity(B, T, D):
    q, k, _, qs, ks = ops.qkv_proj(spec_of(T, D), rnd(B, T, D, seed=1), rnd(3, D, D, seed=2, scale=D ** -0.5))
    return lambda: torch.cat([t.view(-1).view(torch.int32) for t in ops.sim_topk(spec_of(T, D), q, k, qs, ks)])


def _linear(M, N, K, **kw):
    a, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    return lambda: ops.linear(a, w, **kw)


def _prenorm_mlp(M):
    x, mom, wf, wx, w2, b2 = _mlp(M)
    return lambda: ops.prenorm_mlp(x, mom, 1e-5, wf, wx, w2, b2)[0]


def _prenorm_linear(M):
    x, mom, wf, wx, _, _ = _mlp(M)
    return lambda: ops.prenorm_linear(x, mom, 1e-5, wf, wx, gelu=True)


# One CTA that takes longer than the limit of the kernels' polling waits (250 ms) and lets its successor start at once, on the
# SMs it leaves idle: a role that polled for what comes after the predecessor would give up, and its output stay unwritten.
@pytest.mark.parametrize("after", [
    lambda: _linear(300, 192, 192), lambda: _linear(300, 768, 768), lambda: _linear(50432, 192, 192), lambda: _linear(25216, 3072, 768),
    lambda: _prenorm_linear(1000), lambda: _prenorm_mlp(300), lambda: _prenorm_mlp(50432), lambda: _similarity(1, 197, 192),
    lambda: _similarity(64, 300, 192), lambda: _similarity(2, 2048, 64)])
def test_waits_start_behind_the_predecessor(after):
    call = after()
    want = call().clone()
    row = torch.zeros(1, 1 << 30, device=DEV, dtype=BF)
    torch.cuda.synchronize()
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e[0].record()
    ops.row_moments(row)
    e[1].record()
    torch.cuda.synchronize()
    assert e[0].elapsed_time(e[1]) > 300
    ops.row_moments(row)                          # (no event in between: the next launch follows it directly)
    got = call()
    torch.cuda.synchronize()
    assert _capi.device_status() == 0
    assert torch.equal(got, want)


def write_linear(out, a, w):
    """out := a @ w.T by the library's GEMM, into a given buffer."""
    (M, K), N = a.shape, w.shape[0]
    assert out.is_contiguous() and out.numel() == M * N
    _capi.check(_capi.lib().convnn_b200_linear(_capi.BF16, a.data_ptr(), K, w.data_ptr(), None, None, 0, out.data_ptr(), N,
                                               M, N, K, 0, ops._stream(a)))


def _weights_of(name):
    """(buffer that a call reads as weights or bias, the call)."""
    if name.startswith("linear"):
        M, N, K = {"linear, few chunks": (300, 192, 192), "linear, many chunks": (300, 768, 768),
                   "linear, resident": (50432, 192, 192), "linear, pair": (25216, 3072, 768),
                   "linear, bias": (300, 192, 192), "linear, bias of a pair": (25216, 3072, 768)}[name]
        a, w, b = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5), rnd(N, seed=3)
        return (b if "bias" in name else w), lambda: ops.linear(a, w, b)
    if name.startswith("prenorm"):
        x, mom, wf, wx, w2, b2 = _mlp(300)
        buf = {"prenorm_linear": wf, "prenorm_linear, extra rows": wx, "prenorm_mlp, w1": wf, "prenorm_mlp, extra rows": wx,
               "prenorm_mlp, w2": w2, "prenorm_mlp, b2": b2}[name]
        if name.startswith("prenorm_linear"):
            return buf, lambda: ops.prenorm_linear(x, mom, 1e-5, wf, wx, gelu=True)
        return buf, lambda: ops.prenorm_mlp(x, mom, 1e-5, wf, wx, w2, b2)[0]
    x = rnd(2, 197, 192, seed=1)
    if name == "softmax_attention":
        w, wo = rnd(576, 192, seed=2, scale=0.07), rnd(192, 192, seed=3, scale=0.07)
        return w, lambda: ops.softmax_attention(x, w, wo, 3)
    if name == "conv1d_attention":
        w, wo, b = rnd(192, 192, seed=2, scale=0.07), rnd(192, 192, seed=3, scale=0.07), rnd(192, seed=4)
        wc, bc = rnd(64, 9, 64, seed=5, scale=0.05), rnd(64, seed=6)
        return w, lambda: ops.conv1d_attention(x, w, b, wc, bc, wo, b, 3, 9)
    if name == "out_proj":
        o, w = rnd(2, 1, 197, 192, seed=2), rnd(192, 192, seed=3, scale=0.07)
        return w, lambda: ops.out_proj(spec_of(197, 192), o, w)
    w, wc, wo = rnd(3, 192, 192, seed=2, scale=0.07), rnd(9, 192, seed=3), rnd(192, 192, seed=4, scale=0.07)
    if name == "qkv_proj":
        return w, lambda: torch.cat(ops.qkv_proj(spec_of(197, 192), x, w)[:3], dim=1)
    return {"forward, w_qkv": w, "forward, taps": wc, "forward, w_o": wo}[name], \
        lambda: ops.forward(spec_of(197, 192), x, (w, wc, None, wo))


# The first kernel of a call reads no weights before its predecessor has ended, which may be the kernel that writes them: a GEMM
# of a few tiles and many chunks, which lets its successor start at once and stores its results at its end.
@pytest.mark.parametrize("name", [
    "linear, few chunks", "linear, many chunks", "linear, resident", "linear, pair", "linear, bias", "linear, bias of a pair",
    "prenorm_linear", "prenorm_linear, extra rows", "prenorm_mlp, w1", "prenorm_mlp, extra rows", "prenorm_mlp, w2", "prenorm_mlp, b2",
    "softmax_attention", "conv1d_attention", "out_proj", "qkv_proj", "forward, w_qkv", "forward, taps", "forward, w_o"])
def test_weights_written_by_the_launch_before_a_call(name):
    buf, call = _weights_of(name)
    n = 16 if name.endswith("extra rows") else buf.shape[-1]
    rows = buf.numel() // n
    R = 16384
    source = [rnd(rows, R, seed=20 + i, scale=R ** -0.5 * n ** -0.5) for i in range(2)]
    mix = rnd(n, R, seed=30)
    want = []
    for a in source:
        write_linear(buf, a, mix)
        torch.cuda.synchronize()
        want.append(call().clone())
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    got = []
    for turn in range(8):
        write_linear(buf, source[turn % 2], mix)
        got.append(call())
    torch.cuda.synchronize()
    assert _capi.device_status() == 0
    assert all(torch.equal(y, want[turn % 2]) for turn, y in enumerate(got))
