"""The other halves of the branching wrappers on the GPU, through the C ABI, against the CPU
oracle: softmax attention (reference layers.py:105-130) and Conv1d attention (layers.py:477-500).

Tolerances: float32 1e-4 relative; bfloat16 2e-2 relative against the float32 oracle on the
same bfloat16-rounded inputs and weights.
"""
import math

import pytest
import torch

import convnn_b200
from convnn_b200 import _capi, ops
from oracle.convnn_oracle import bf16_round, conv1d_attention, softmax_attention
from gpu_util import DEV, launches, on_148_sms, rel_err

pytestmark = pytest.mark.gpu


def _uni(shape, fan_in, g):
    return (torch.rand(shape, generator=g) * 2 - 1) / math.sqrt(fan_in)


ATTN_CASES = [
    # B, T, D, H, dtype          (bfloat16 with T <= 256 and d_k % 16 == 0: the tensor-core kernel)
    (2, 197, 384, 12, torch.bfloat16),      # the ViT-Base BranchAttention half: d_k = 32
    (3, 197, 96, 3, torch.bfloat16),
    (2, 65, 48, 3, torch.bfloat16),         # d_k = 16, one row tile
    (1, 256, 128, 1, torch.bfloat16),       # d_k = 128, full 256-token tile
    (2, 130, 192, 2, torch.bfloat16),       # d_k = 96: three 32-channel chunks
    (2, 300, 64, 2, torch.bfloat16),        # more than 256 tokens: SIMT kernel
    (2, 197, 96, 3, torch.float32),
    (2, 40, 40, 2, torch.float32),          # d_k = 20
]


@pytest.mark.parametrize("B,T,D,H,dtype", ATTN_CASES)
def test_softmax_attention_matches_oracle(B, T, D, H, dtype):
    g = torch.Generator().manual_seed(B * 100 + T + D)
    w = {f"W_{n}.weight": _uni((D, D), D, g) * (3.0 if n in "qk" else 1.0) for n in "qkvo"}
    x = torch.randn(B, T, D, generator=g)
    if dtype == torch.bfloat16:
        w = {k: bf16_round(v) for k, v in w.items()}
        x = bf16_round(x)
    m = convnn_b200.MultiHeadAttention(D, H, 0.0)
    m.load_state_dict(w, strict=True)
    m = m.eval().to(DEV, dtype)
    with torch.no_grad():
        y = m(x.to(DEV, dtype))
        # channel-slice input and output, as MultiHeadBranchingAttention uses it
        wide = torch.zeros(B, T, D + 16, device=DEV, dtype=dtype)
        wide[:, :, 16:] = x.to(DEV, dtype)
        dst = torch.full((B, T, D + 24), 5.0, device=DEV, dtype=dtype)
        m(wide[:, :, 16:], out=dst[:, :, 8:8 + D])
    torch.cuda.synchronize()
    assert _capi.device_status() == 0
    want = softmax_attention(x, w, H)
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    assert rel_err(y, want) < tol
    assert torch.equal(dst[:, :, 8:8 + D], y)
    assert bool((dst[:, :, :8] == 5.0).all()) and bool((dst[:, :, 8 + D:] == 5.0).all())


CONV_CASES = [
    # B, T, D, H, kernel_size, dtype
    (2, 197, 96, 3, 9, torch.bfloat16),     # d_k = 32: the fused convolution
    (2, 197, 48, 3, 5, torch.bfloat16),     # d_k = 16
    (2, 197, 384, 12, 9, torch.bfloat16),
    (2, 65, 40, 1, 4, torch.bfloat16),      # d_k = 40 (SIMT kernel), even kernel size
    (2, 197, 96, 3, 9, torch.float32),
    (3, 65, 24, 1, 4, torch.float32),
    (2, 33, 32, 2, 1, torch.float32),
]


@pytest.mark.parametrize("B,T,D,H,ks,dtype", CONV_CASES)
def test_conv1d_attention_matches_oracle(B, T, D, H, ks, dtype):
    g = torch.Generator().manual_seed(B * 100 + T + D + ks)
    dk = D // H
    w = {"W_x.weight": _uni((D, D), D, g), "W_x.bias": _uni((D,), D, g),
         "conv.weight": _uni((dk, dk, ks), dk * ks, g), "conv.bias": _uni((dk,), dk * ks, g),
         "W_o.weight": _uni((D, D), D, g), "W_o.bias": _uni((D,), D, g)}
    x = torch.randn(B, T, D, generator=g)
    if dtype == torch.bfloat16:
        w = {k: bf16_round(v) for k, v in w.items()}
        x = bf16_round(x)
    m = convnn_b200.MultiHeadConv1dAttention(D, H, ks)
    m.load_state_dict(w, strict=True)
    m = m.eval().to(DEV, dtype)
    with torch.no_grad():
        y = m(x.to(DEV, dtype))
        y2 = m(x.to(DEV, dtype))
    torch.cuda.synchronize()
    assert _capi.device_status() == 0
    assert torch.equal(y, y2)
    want = conv1d_attention(x, w, H, ks)
    assert rel_err(y, want) < (1e-4 if dtype == torch.float32 else 2e-2)


# The fused convolution: one token, whole and ragged 128-row tiles, even kernels, several slices per CTA, heads of 64, one set
# of taps in flight (250 tokens); then three that are unfolded (257 tokens: another tile; 25 taps: they do not fit).
@pytest.mark.parametrize("B,T,D,H,ks", [(2, 1, 32, 1, 3), (1, 128, 64, 2, 8), (60, 129, 96, 3, 9), (200, 65, 32, 2, 4),
                                        (2, 50, 128, 2, 1), (2, 250, 64, 1, 5), (1, 257, 64, 1, 5), (2, 300, 32, 1, 25), (1, 60, 64, 1, 25)])
def test_fused_conv1d_attention_matches_oracle(B, T, D, H, ks):
    test_conv1d_attention_matches_oracle(B, T, D, H, ks, torch.bfloat16)


# Which shapes the fused convolution takes (slices of at most two tiles, few tiles, or many slices; not many tiny sequences) and
# its result there and beside them: y = x and out = (conv, reinterpreted) by products with the identity, every element
# bounded.  Kernels of 16 channels up to 32 taps (the widest mask), one set of taps in flight (250 x 64 x 5, 130 x 32 x 15),
# whole and ragged tiles, ends of the sequence with even kernels.
@on_148_sms
@pytest.mark.parametrize("B,T,H,dk,ks,fused", [
    (1, 1000, 1, 32, 9, False), (1, 4096, 1, 16, 9, False), (1, 600, 1, 64, 1, False), (25, 600, 1, 16, 25, False),
    (32, 1000, 1, 64, 3, False), (400, 9, 3, 32, 9, False), (300, 17, 1, 32, 15, False), (2, 300, 1, 32, 25, False),
    (2, 300, 1, 16, 25, False), (2, 257, 1, 64, 5, False), (1, 300, 1, 32, 9, True), (8, 1000, 1, 16, 5, True), (16, 1000, 2, 32, 9, True), (25, 300, 6, 32, 9, True),
    (2, 128, 1, 16, 32, True), (2, 130, 2, 32, 15, True), (3, 256, 1, 16, 17, True), (2, 250, 1, 64, 5, True), (1, 127, 2, 64, 4, True),
    (60, 129, 5, 32, 8, True), (148, 9, 1, 64, 9, True)])
def test_fused_conv1d_every_element(B, T, H, dk, ks, fused):
    D, left = H * dk, (ks - 1) // 2
    g = torch.Generator(device=DEV).manual_seed(T + ks)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    eye, zero = torch.eye(D, device=DEV).bfloat16(), torch.zeros(D, device=DEV).bfloat16()
    x, w, b = rnd(B, T, D), rnd(dk, ks, dk), rnd(dk)
    call = lambda: ops.conv1d_attention(x, eye, zero, w, b, eye, zero, H, ks)
    assert any("conv1d_tc_kernel" in n for n in launches(call)) == fused
    got = call().double()
    torch.cuda.synchronize()
    assert _capi.device_status() == 0
    y = torch.nn.functional.pad(x.double().view(B, T, H, dk).permute(0, 2, 1, 3), (0, 0, left, ks - 1 - left))
    z, mass = [t.expand(B, H, T, dk).clone() for t in (b.double(), b.double().abs())]
    for j in range(ks):
        z += y[:, :, j:j + T] @ w[:, j].double().T
        mass += y[:, :, j:j + T].abs() @ w[:, j].double().abs().T
    flat = lambda t: t.reshape(B, H, dk, T).permute(0, 3, 1, 2).reshape(B, T, D)       # (t, c) rows read back as (c, t)
    # fp32 sums of ks * dk terms, one rounding of the result (the products with the identity are exact)
    bound = (ks * dk + 8) * 2.0 ** -24 * flat(mass) + 2.0 ** -8 * flat(z).abs() + 1e-30
    assert bool(((got - flat(z)).abs() <= bound).all())


def test_branching_modules_fold_the_skip_connection():
    """residual + layer(x) from one call equals the two-step result bit for bit."""
    g = torch.Generator().manual_seed(5)
    x = torch.randn(2, 197, 96, generator=g).to(DEV, torch.bfloat16)
    for m in (convnn_b200.MultiHeadBranchingAttention(96, 3, 0.0, 9, "all", -1, 0, "cosine", 197, False, "standard"),
              convnn_b200.MultiHeadBranchingConv(96, 3, 0.0, 5, 9, "all", -1, 0, "cosine")):
        m = m.eval().to(DEV, torch.bfloat16)
        with torch.no_grad():
            y = m(x)
            z = m(x, residual=x)
        assert torch.equal(z, x + y)


# Off the tensor cores: ends of the 16- and 32-row tiles, of the chunks of 32 channels and 128 keys, channels that are no multiple of
# eight, several passes over the keys, a sequence whose scores no tile has room for.
@pytest.mark.parametrize("B,T,D,H,dtype", [
    (2, 1, 8, 1, torch.float32), (2, 15, 33, 1, torch.float32), (1, 129, 60, 2, torch.float32), (3, 65, 192, 1, torch.bfloat16),
    (1, 128, 384, 1, torch.bfloat16), (2, 257, 136, 1, torch.bfloat16), (40, 257, 64, 2, torch.bfloat16), (50, 197, 160, 1, torch.float32),
    (1, 7000, 16, 1, torch.float32), (60, 197, 48, 1, torch.float32), (1, 33, 30, 2, torch.bfloat16)])
def test_softmax_attention_tiles(B, T, D, H, dtype):
    g = torch.Generator().manual_seed(T + D)
    w = {f"W_{n}.weight": _uni((D, D), D, g) * (3.0 if n in "qk" else 1.0) for n in "qkvo"}
    x = torch.randn(B, T, D, generator=g)
    if dtype == torch.bfloat16:
        w = {n: bf16_round(t) for n, t in w.items()}
        x = bf16_round(x)
    w_qkv = torch.stack([w[f"W_{n}.weight"] for n in "qkv"]).to(DEV, dtype)
    x_dev, w_o = x.to(DEV, dtype), w["W_o.weight"].to(DEV, dtype)
    call = lambda: ops.softmax_attention(x_dev, w_qkv, w_o, H)
    assert any("attention_tile_kernel" in n for n in launches(call)) == (T < 6000)
    assert rel_err(call(), softmax_attention(x, w, H)) < (1e-4 if dtype == torch.float32 else 2e-2)


# Short sequences of many heads: a warp per row; the same sequences by themselves: a tile of rows.  Both give the same bits.
@on_148_sms
@pytest.mark.parametrize("B,T,D,H,few,dtype", [
    (4854, 2, 8, 1, 16, torch.bfloat16), (500, 7, 192, 3, 2, torch.float32), (1500, 9, 48, 2, 2, torch.bfloat16),
    (700, 11, 24, 1, 16, torch.float32), (800, 20, 8, 1, 16, torch.float32), (1000, 1, 40, 1, 16, torch.float32)])
def test_softmax_attention_of_short_sequences(B, T, D, H, few, dtype):
    g = torch.Generator().manual_seed(T + D)
    w = {f"W_{n}.weight": _uni((D, D), D, g) * (3.0 if n in "qk" else 1.0) for n in "qkvo"}
    x = torch.randn(B, T, D, generator=g)
    if dtype == torch.bfloat16:
        w = {n: bf16_round(t) for n, t in w.items()}
        x = bf16_round(x)
    w_qkv = torch.stack([w[f"W_{n}.weight"] for n in "qkv"]).to(DEV, dtype)
    x_dev, w_o = x.to(DEV, dtype), w["W_o.weight"].to(DEV, dtype)
    call = lambda n=B: ops.softmax_attention(x_dev[:n], w_qkv, w_o, H)
    assert any("attention_simt_kernel" in n for n in launches(call))
    got = call()
    assert rel_err(got[:64], softmax_attention(x[:64], w, H)) < (1e-4 if dtype == torch.float32 else 2e-2)
    if T > 8 or T == 1:
        assert any("attention_tile_kernel" in n for n in launches(lambda: call(few)))
        assert torch.equal(call(few), got[:few])
