"""Similarity of bfloat16 heads at widths that do not fill the tensor-core kernels' 64-channel chunks (zero-filled by the
copies) or are no multiple of sixteen (fp32 pipes): lists against float64 on the same bfloat16 q and k."""
import pytest
import torch

from convnn_b200 import ops
from gpu_util import DEV

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("T,S,H,dk,coord", [(130, 130, 1, 8, False), (65, 65, 2, 24, False), (197, 40, 4, 48, False), (257, 257, 1, 96, False),
                                            (577, 150, 1, 384, True), (65, 65, 3, 64, True), (70, 33, 1, 15, True),
                                            (1100, 1100, 1, 104, False), (1030, 1025, 1, 384, True)])
@pytest.mark.parametrize("K", [5, 9, 16])
def test_lists(T, S, H, dk, coord, K):
    g = torch.Generator(device=DEV).manual_seed(T + dk)
    B = 2
    mode = "all" if S == T else "spatial"
    spec = ops.LayerSpec(H * dk, H, K, mode, "cosine", "standard" if coord else "depthwise", True, coord, T)
    C = dk + int(coord)
    Cp = (C + 7) // 8 * 8 if coord else dk
    q, k = (torch.zeros(B, n, H, Cp, device=DEV) for n in (S, T))
    q[..., :C] = torch.randn(B, S, H, C, device=DEV, generator=g)
    k[..., :C] = torch.randn(B, T, H, C, device=DEV, generator=g)
    q, k = q.to(torch.bfloat16), k.to(torch.bfloat16)
    qs, ks = (1 / t.float().norm(dim=-1).permute(0, 2, 1).contiguous() for t in (q, k))
    cand = None if S == T else torch.arange(S, device=DEV, dtype=torch.int32) * (T // S)
    idx, val = ops.sim_topk(spec, q, k, qs, ks, cand)
    sim = torch.einsum("bthc,bshc->bhts", k.double(), q.double()) * ks.double().unsqueeze(-1) * qs.double().unsqueeze(2)
    if cand is not None:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        sim = sim.masked_fill(own, -0.1)
    n = K if cand is None else K - 1
    want = sim.topk(n, -1).values
    # |key| <= 1: the n-th best value moves by no more than the rounding of a C-term fp32 dot product of unit vectors
    assert float((val[..., K - n:].double() - want).abs().max()) <= (C + 16) * EPS
    got = idx[..., K - n:].long()
    col = got if cand is None else got // (T // S)
    picked = torch.gather(sim, -1, col)
    assert float((picked - val[..., K - n:].double()).abs().max()) <= (C + 16) * EPS      # values belong to their indices


@pytest.mark.parametrize("T,S,H,dk", [(577, 150, 1, 384), (197, 197, 3, 64), (130, 33, 1, 768), (1100, 1100, 1, 192), (65, 65, 2, 16)])
@pytest.mark.parametrize("metric", ["cosine", "matmul", "euclidean"])
def test_coordinate_channel_keeps_the_fp32_sums(T, S, H, dk, metric):
    """Products of bfloat16 values are exact in float32, so the sums over the stored channels have to be those of the
    float32 path on the same values, bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(T + dk)
    K, C = 9, dk + 1
    spec = ops.LayerSpec(H * dk, H, K, "all" if S == T else "spatial", metric, "standard", True, True, T)
    q, k = (torch.zeros(2, n, H, (C + 7) // 8 * 8, device=DEV) for n in (S, T))
    q[..., :C] = torch.randn(2, S, H, C, device=DEV, generator=g)
    k[..., :C] = torch.randn(2, T, H, C, device=DEV, generator=g)
    q, k = q.to(torch.bfloat16), k.to(torch.bfloat16)
    n2 = [t.float().pow(2).sum(-1).permute(0, 2, 1).contiguous() for t in (q, k)]
    qs, ks = [t.rsqrt() for t in n2] if metric == "cosine" else n2
    cand = None if S == T else torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32)
    got, want = (ops.sim_topk(spec, a, b, qs, ks, cand) for a, b in ((q, k), (q.float(), k.float())))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("C", [64, 96, 144, 272])
@pytest.mark.parametrize("K", [9, 16, 17])
def test_long_sequences_give_the_same_lists_in_batches_of_any_size(C, K):
    """Which of the two long-sequence kernels runs depends on the number of rows: one, two, five and nine rounds of it."""
    g = torch.Generator(device=DEV).manual_seed(C)
    T = 1024
    spec = ops.LayerSpec(C, 1, K, "all", "cosine", "depthwise", True, False, T)
    q, k = (torch.randn(160, T, 1, C, device=DEV, generator=g).bfloat16() for _ in range(2))
    qs, ks = (1 / t.float().norm(dim=-1).permute(0, 2, 1).contiguous() for t in (q, k))
    want = ops.sim_topk(spec, q, k, qs, ks)
    for B in (1, 33, 80):
        got = ops.sim_topk(spec, q[:B], k[:B], qs[:B].contiguous(), ks[:B].contiguous())
        assert torch.equal(got[0], want[0][:B]) and torch.equal(got[1], want[1][:B])
