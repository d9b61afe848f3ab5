"""Depthwise gather / conv at the edges of its tiles (tokens per CTA, tokens per thread, channel groups, weights that are
not 16-byte rows) and the weighted neighbour block, against float64."""
import pytest
import torch

from convnn_b200 import ops
from gpu_util import DEV, launches, on_148_sms

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("B,T,H,dk,K", [(1, 1, 1, 8, 1), (1, 65, 1, 768, 16), (3, 197, 3, 32, 9), (2, 300, 1, 40, 32), (9, 513, 2, 64, 5),
                                        (40, 1025, 1, 64, 9), (33, 1024, 4, 16, 25), (1, 13, 1, 264, 7)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("metric,softmax", [("cosine", True), ("euclidean", True), ("euclidean", False), ("matmul", False)])
def test_depthwise_against_float64(B, T, H, dk, K, dtype, metric, softmax):
    g = torch.Generator(device=DEV).manual_seed(B * T + K)
    spec = ops.LayerSpec(H * dk, H, K, "all", metric, "depthwise", softmax, False, T)
    v = torch.randn(B, T, H, dk, device=DEV, generator=g).to(dtype)
    idx = torch.randint(0, T, (B, H, T, K), device=DEV, generator=g, dtype=torch.int32)
    val = torch.rand(B, H, T, K, device=DEV, generator=g) + 0.25
    w = torch.randn(K, dk, device=DEV, generator=g).to(dtype)
    got = ops.gather_conv(spec, v, idx, val, w)
    x = val.double() * (1 if metric != "euclidean" else -1)
    p = torch.softmax(x, -1) if softmax else (val.double() if metric != "euclidean" else 1 / (val.double() + 1e-8))
    rows = v.double().permute(0, 2, 1, 3)
    want, mass = torch.zeros(B, H, T, dk, device=DEV, dtype=torch.double), torch.zeros(B, H, T, dk, device=DEV, dtype=torch.double)
    for j in range(K):
        term = p[..., j:j + 1] * torch.gather(rows, 2, idx[..., j:j + 1].long().expand(B, H, T, dk)) * w[j].double()
        want += term
        mass += term.abs()
    bound = (2 * K + 24) * EPS * mass + (0 if dtype == torch.float32 else 2.0 ** -8) * want.abs() + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("B,T,H,dk,K", [(2, 65, 1, 768, 25), (1, 3, 1, 16, 1), (5, 197, 12, 32, 9), (2, 1030, 1, 192, 5)])
def test_standard_conv_bfloat16_against_float64(B, T, H, dk, K):
    g = torch.Generator(device=DEV).manual_seed(T)
    spec = ops.LayerSpec(H * dk, H, K, "all", "cosine", "standard", True, False, T)
    v = torch.randn(B, T, H, dk, device=DEV, generator=g).to(torch.bfloat16)
    idx = torch.randint(0, T, (B, H, T, K), device=DEV, generator=g, dtype=torch.int32)
    val = torch.randn(B, H, T, K, device=DEV, generator=g)
    w = (torch.randn(dk, K, dk, device=DEV, generator=g) / (K * dk) ** 0.5).to(torch.bfloat16)
    got = ops.gather_conv(spec, v, idx, val, w)
    p = torch.softmax(val.double(), -1)
    rows = v.double().permute(0, 2, 1, 3)
    want, mass = torch.zeros(B, H, T, dk, device=DEV, dtype=torch.double), torch.zeros(B, H, T, dk, device=DEV, dtype=torch.double)
    for j in range(K):
        nb = p[..., j:j + 1] * torch.gather(rows, 2, idx[..., j:j + 1].long().expand(B, H, T, dk))
        want += nb @ w[:, j].double().T
        mass += nb.abs() @ w[:, j].double().abs().T
    # the weighted block is rounded to bfloat16 once, the result once; fp32 sums of K * dk terms
    bound = (2.0 ** -9 + (K * dk + 16) * EPS) * mass + 2.0 ** -8 * want.abs() + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


# Selection and depthwise conv in one kernel (few rows per SM, at most 17 neighbours) against the two stages, whose lists and
# sums are the same: bit for bit.  One row, ragged sequences, sixteen and seventeen neighbours, one channel group, the widest
# taps, several heads, every way of weighting; then two rows per warp (32 rows per CTA), odd ends and seventeen neighbours among
# them.  The last four do not go to it: too many rows per CTA, ranges across heads, and long taps over short lists.
@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk,K,fused", [
    (1, 1, 1, 1, 16, 1, True), (3, 197, 197, 1, 192, 9, True), (1, 197, 197, 3, 64, 9, True), (2, 65, 40, 1, 48, 17, True),
    (5, 130, 100, 1, 16, 16, True), (2, 257, 225, 1, 384, 5, True), (1, 33, 33, 2, 80, 12, True), (1, 500, 256, 1, 768, 10, True),
    (16, 197, 197, 1, 64, 9, True), (20, 197, 197, 1, 192, 9, True), (10, 200, 150, 2, 32, 17, True), (40, 83, 60, 1, 16, 17, True),
    (139, 17, 17, 1, 32, 9, True), (6, 250, 250, 3, 32, 16, True),
    (40, 197, 197, 1, 64, 9, False), (200, 17, 17, 1, 32, 9, False), (300, 9, 9, 1, 16, 9, False), (23, 100, 100, 1, 768, 9, False)])
@pytest.mark.parametrize("metric,softmax", [("cosine", True), ("matmul", False), ("euclidean", True), ("euclidean", False)])
def test_selection_with_conv_equals_the_stages(B, T, S, H, dk, K, fused, metric, softmax):
    D = H * dk
    g = torch.Generator(device=DEV).manual_seed(T + S + K)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    spec = ops.LayerSpec(D, H, K, "spatial" if S != T else "all", metric, "depthwise", softmax, False, T)
    x, w_qkv, w_o, taps = rnd(B, T, D), rnd(3, D, D) * D ** -0.5, rnd(D, D) * D ** -0.5, rnd(K, dk)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if S != T else None
    names = launches(lambda: ops.forward(spec, x, (w_qkv, taps, None, w_o), cand))
    assert any("sim_topk_rows_kernel" in n and "Lb1E" in n for n in names) == fused
    whole = ops.forward(spec, x, (w_qkv, taps, None, w_o), cand)
    q, k, v, qs, ks = ops.qkv_proj(spec, x, w_qkv, cand)
    idx, val = ops.sim_topk(spec, q, k, qs, ks, cand)
    out = ops.out_proj(spec, ops.gather_conv(spec, v, idx, val, taps, None, S=S), w_o, S=S)
    assert torch.equal(whole.isnan(), out.isnan()) and torch.equal(whole.nan_to_num(), out.nan_to_num())


# The standard conv whose neighbour block stays on the SM: edges of its 128-token tiles, of a producer warp's eight tokens and of
# its groups of taps, the longest lists, several slices per CTA; from the eleventh on shapes
# that others take: few or sparse tiles, taps that do not fit, 24 channels.
@pytest.mark.parametrize("B,T,H,dk,K", [(1, 127, 2, 16, 5), (2, 128, 1, 32, 6), (148, 129, 1, 64, 3), (3, 9, 2, 64, 4), (120, 256, 1, 32, 32),
                                        (100, 197, 3, 32, 9), (74, 300, 2, 16, 17), (148, 250, 4, 16, 17), (148, 300, 1, 32, 9), (148, 256, 1, 64, 9),
                                        (1, 129, 3, 64, 3), (2, 256, 1, 32, 32), (60, 137, 3, 32, 9), (80, 300, 2, 16, 17), (2, 300, 1, 32, 9),
                                        (1, 40, 2, 64, 25), (2, 50, 2, 24, 9)])
def test_standard_conv_tiles(B, T, H, dk, K):
    test_standard_conv_bfloat16_against_float64(B, T, H, dk, K)


# Which shapes it takes, one head (the stage) and several (a layer's reinterpreted store): one tile per CTA, two, several; full
# and sparse tiles; few and many taps.
@on_148_sms
@pytest.mark.parametrize("B,T,H,dk,K,fused", [
    (8, 65, 1, 32, 9, True), (148, 100, 1, 64, 9, True), (1, 128, 1, 16, 32, True), (8, 197, 1, 64, 9, False), (74, 256, 1, 64, 5, False),
    (32, 256, 1, 32, 16, False), (148, 130, 1, 64, 3, True), (100, 197, 1, 32, 3, True), (148, 600, 1, 16, 5, True), (200, 100, 1, 16, 9, True),
    (600, 17, 1, 32, 9, False), (600, 197, 1, 64, 5, False), (600, 197, 1, 32, 9, True), (300, 256, 1, 16, 16, False), (200, 65, 1, 16, 25, True),
    (1, 600, 1, 32, 9, False), (1, 40, 1, 64, 25, False), (1, 40, 1, 24, 9, False)])
def test_standard_conv_routes(B, T, H, dk, K, fused):
    g = torch.Generator(device=DEV).manual_seed(T)
    spec = ops.LayerSpec(H * dk, H, K, "all", "cosine", "standard", True, False, T)
    v = torch.randn(B, T, H, dk, device=DEV, generator=g).bfloat16()
    idx = torch.randint(0, T, (B, H, T, K), device=DEV, generator=g, dtype=torch.int32)
    val, w = torch.randn(B, H, T, K, device=DEV, generator=g), torch.randn(dk, K, dk, device=DEV, generator=g).bfloat16()
    assert any("conv_std_tc_kernel" in n for n in launches(lambda: ops.gather_conv(spec, v, idx, val, w))) == fused
    test_standard_conv_bfloat16_against_float64(B, T, H, dk, K)


@on_148_sms
@pytest.mark.parametrize("B,T,H,dk,K,fused", [(2, 197, 3, 32, 9, True), (2, 65, 2, 64, 9, True), (1, 130, 4, 16, 5, True), (1, 197, 3, 64, 3, True),
                                              (60, 137, 3, 32, 9, True), (74, 197, 2, 64, 9, True), (40, 300, 4, 32, 9, True),
                                              (3, 65, 2, 64, 16, False), (4, 256, 2, 64, 9, False), (300, 17, 2, 16, 9, False)])
@pytest.mark.parametrize("metric,softmax", [("cosine", True), ("matmul", False), ("euclidean", True), ("euclidean", False)])
def test_standard_conv_in_the_flat_reinterpretation(B, T, H, dk, K, fused, metric, softmax):
    """The layer's call, whose conv stores the reinterpreted rows, against the stages, which store them as they are."""
    D = H * dk
    g = torch.Generator(device=DEV).manual_seed(T + K)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    spec = ops.LayerSpec(D, H, K, "all", metric, "standard", softmax, False, T)
    x, w_qkv, w_o, taps = rnd(B, T, D), rnd(3, D, D) * D ** -0.5, rnd(D, D) * D ** -0.5, rnd(dk, K, dk) * (K * dk) ** -0.5
    names = launches(lambda: ops.forward(spec, x, (w_qkv, taps, None, w_o), None))
    assert [any(k in n for n in names) for k in ("conv_std_tc_kernel", "merge_heads_kernel")] == [fused, not fused]
    whole = ops.forward(spec, x, (w_qkv, taps, None, w_o), None)
    q, k, v, qs, ks = ops.qkv_proj(spec, x, w_qkv, None)
    idx, val = ops.sim_topk(spec, q, k, qs, ks, None)
    out = ops.out_proj(spec, ops.gather_conv(spec, v, idx, val, taps), w_o, S=T)
    assert torch.equal(whole.isnan(), out.isnan()) and torch.equal(whole.nan_to_num(), out.nan_to_num())


# Four tokens per thread: a last set of one, two, three tokens, one tap and many, taps and rows of one vector less than a warp's.
@pytest.mark.parametrize("B,T,H,dk,K", [(1, 6401, 1, 384, 9), (2, 3203, 1, 384, 1), (5, 1283, 1, 384, 25), (3, 1024, 2, 248, 5), (1, 40001, 1, 72, 32)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_sets_of_four_tokens(B, T, H, dk, K, dtype):
    test_depthwise_against_float64(B, T, H, dk, K, dtype, "cosine", True)
    test_depthwise_against_float64(B, T, H, dk, K, dtype, "euclidean", False)


# Every form by the rounds of CTAs per SM (tokens per thread, taps in flight, CTAs per SM that fit), as the dispatch picks them.
@on_148_sms
@pytest.mark.parametrize("B,T,H,dk,K,dtype,form", [
    (3, 33, 1, 64, 9, torch.float32, "1, 4, 4"), (71, 34, 2, 128, 3, torch.float32, "1, 2, 5"), (9, 701, 2, 64, 5, torch.float32, "1, 2, 6"),
    (12, 158, 1, 768, 5, torch.float32, "4, 2, 2"), (7, 3098, 2, 96, 9, torch.float32, "4, 1, 3"), (2, 473, 12, 128, 3, torch.bfloat16, "1, 2, 5"),
    (5, 660, 1, 256, 9, torch.bfloat16, "1, 4, 4"), (10, 1611, 3, 96, 25, torch.bfloat16, "4, 2, 2"), (76, 518, 6, 16, 3, torch.bfloat16, "4, 2, 2"),
    (40, 1024, 4, 16, 25, torch.bfloat16, "4, 1, 3")])
def test_forms_of_the_depthwise_gather(B, T, H, dk, K, dtype, form):
    spec = ops.LayerSpec(H * dk, H, K, "all", "cosine", "depthwise", True, False, T)
    v, w = torch.zeros(B, T, H, dk, device=DEV, dtype=dtype), torch.zeros(K, dk, device=DEV, dtype=dtype)
    idx, val = torch.zeros(B, H, T, K, device=DEV, dtype=torch.int32), torch.zeros(B, H, T, K, device=DEV)
    name, = launches(lambda: ops.gather_conv(spec, v, idx, val, w))
    assert "gather_conv_dw_kernel" in name and "Li{}ELi{}ELi{}EE".format(*form.split(", ")) in name
    test_depthwise_against_float64(B, T, H, dk, K, dtype, "cosine", True)
    test_depthwise_against_float64(B, T, H, dk, K, dtype, "euclidean", False)


# Grids that leave SMs idle: one to a few tokens per CTA, a ragged last one, eight taps in flight with 13, 16 and 25 of them.
@pytest.mark.parametrize("B,T,H,dk,K", [(1, 13, 1, 8, 13), (2, 65, 1, 96, 25), (1, 297, 1, 192, 16), (1, 593, 1, 64, 25), (3, 197, 3, 64, 32)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_small_grids(B, T, H, dk, K, dtype):
    test_depthwise_against_float64(B, T, H, dk, K, dtype, "cosine", True)
    test_depthwise_against_float64(B, T, H, dk, K, dtype, "euclidean", False)


# Eight taps in flight on small grids only where they leave at most three.
@on_148_sms
@pytest.mark.parametrize("K,form", [(13, "1, 4, 4"), (16, "1, 8, 2"), (19, "1, 8, 2"), (20, "1, 4, 4"), (25, "1, 8, 2"), (31, "1, 4, 4")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_taps_in_flight_on_small_grids(K, form, dtype):
    test_forms_of_the_depthwise_gather(2, 65, 1, 96, K, dtype, form)
