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
