"""Values stored into rows of padded heads (bfloat16, coordinate channel)."""
import pytest
import torch

from convnn_b200 import ops
from gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,dk", [(1, 8), (1, 16), (2, 8), (3, 24), (4, 16), (3, 64), (1, 384), (12, 64)])
@pytest.mark.parametrize("B,T", [(1, 1), (2, 65), (1, 129)])
def test_values(H, dk, B, T):
    g = torch.Generator(device=DEV).manual_seed(H * 100 + dk)
    D = H * dk
    w = [(torch.randn(D, D, device=DEV, generator=g) / D ** 0.5).bfloat16() for _ in range(4)]
    x = torch.randn(B, T, D, device=DEV, generator=g).bfloat16()
    spec = ops.LayerSpec(D, H, 1, "all", "cosine", "standard", True, True, T)
    conv = (torch.zeros(dk, dk + 1, 1, device=DEV),)
    packed = ops.pack_weights(spec, *w, conv, torch.bfloat16, torch.device(DEV))[0]       # W_q, W_k, W_v, W_o
    _, _, v, _, _ = ops.qkv_proj(spec, x, packed)
    want = torch.einsum("btd,nd->btn", x.double(), w[2].double()).view(B, T, H, dk)
    got = v[..., :dk].double()
    # one bfloat16 rounding of the sum, and the fp32 rounding of D terms whose magnitudes add up to S
    s = torch.einsum("btd,nd->btn", x.double().abs(), w[2].double().abs()).view(B, T, H, dk)
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + D * 2.0 ** -24 * s).all())
    line = torch.linspace(-1, 1, T).bfloat16().to(DEV).view(1, T, 1).expand(B, T, H)
    assert torch.equal(v[..., dk], line) and not bool(v[..., dk + 1:].any())


@pytest.mark.parametrize("H,dk", [(1, 384), (3, 64), (2, 24), (1, 768)])
def test_projections_keep_the_fp32_sums(H, dk):
    """Products of bfloat16 values are exact in float32: k, v and q are the float32 path's sums, rounded once."""
    g = torch.Generator(device=DEV).manual_seed(H * 100 + dk)
    D, T = H * dk, 577
    w = [(torch.randn(D, D, device=DEV, generator=g) / D ** 0.5).bfloat16() for _ in range(4)]
    x = torch.randn(4, T, D, device=DEV, generator=g).bfloat16()
    spec = ops.LayerSpec(D, H, 1, "all", "matmul", "standard", True, True, T)
    packed = ops.pack_weights(spec, *w, (torch.zeros(dk, dk + 1, 1, device=DEV),), torch.bfloat16, torch.device(DEV))[0]
    got, want = ops.qkv_proj(spec, x, packed)[:3], ops.qkv_proj(spec, x.float(), packed.float())[:3]
    for a, b in zip(got, want):
        assert torch.equal(a[..., :dk], b[..., :dk].bfloat16())
