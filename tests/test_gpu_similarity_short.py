"""Two-pass selection over at most 256 candidates: integer-valued q and k make every similarity exact in float32, so lists,
their order and the tie rule (lower column first) are compared exactly with a stable sort, ties and NaN included."""
import math

import pytest
import torch

from convnn_b200 import ops
from gpu_util import DEV, launches, on_148_sms

pytestmark = pytest.mark.gpu


def expect(key, n):
    """(rows, S) float32 keys -> the n best columns, ties by column; NaN and -inf are never picked, empty slots hold 0 / -inf."""
    usable = ~key.isnan() & (key > -math.inf)
    ranked = torch.where(usable, key, torch.full_like(key, -math.inf))
    order = torch.sort(ranked, dim=-1, descending=True, stable=True)
    idx = torch.where(order.values[..., :n] > -math.inf, order.indices[..., :n], torch.zeros_like(order.indices[..., :n]))
    return idx, order.values[..., :n]


@pytest.mark.parametrize("T,S,H,dk", [(1, 1, 1, 8), (5, 5, 2, 16), (33, 17, 1, 32), (129, 32, 3, 24), (65, 65, 1, 64), (97, 96, 1, 200),
                                      (300, 127, 1, 64), (128, 128, 2, 32), (129, 129, 1, 64), (197, 197, 3, 64), (197, 197, 1, 192),
                                      (577, 150, 1, 384), (255, 255, 1, 48), (256, 256, 1, 768), (700, 256, 2, 32)])
@pytest.mark.parametrize("K", [1, 4, 5, 9, 11, 16, 24, 25, 32])
@pytest.mark.parametrize("values", ["few", "many", "nan"])
def test_exact_lists(T, S, H, dk, K, values):
    sampled = S != T
    n = K - 1 if sampled else K
    if n < 1 or n > S:
        pytest.skip("list longer than the candidates")
    g = torch.Generator().manual_seed(T * 1000 + S + K)
    B = 3
    top = 1 if values == "few" else 11               # products and sums stay far below 2^24
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), generator=g).float() for r in (S, T))
    if values == "nan":
        q[:, ::3] = math.nan                          # a third of the candidates
        q[1, 2:] = math.nan                           # one image with two candidates left
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, generator=g)[:S].to(torch.int32) if sampled else None
    idx, val = ops.sim_topk(spec, q.bfloat16().to(DEV), k.bfloat16().to(DEV), None, None, None if cand is None else cand.to(DEV))
    key = torch.einsum("bthc,bshc->bhts", k, q)
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32), key)
    want_idx, want_key = expect(key, n)
    want_tok = want_idx if cand is None else cand.long()[want_idx]
    got_idx, got_val = idx.long().cpu()[..., K - n:], val.cpu()[..., K - n:]
    assert torch.equal(got_idx, want_tok)
    real = want_key > -math.inf
    if sampled:
        assert torch.equal(idx.long().cpu()[..., 0], torch.arange(T).expand(B, H, T))
        assert bool((got_val[(want_tok == torch.arange(T).view(1, 1, T, 1)) & real] == -0.1).all())
        real &= want_tok != torch.arange(T).view(1, 1, T, 1)
    want_val = want_key / torch.tensor(math.sqrt(dk), dtype=torch.float32)
    # one division: equal up to its rounding
    assert float(((got_val - want_val)[real].abs() / want_val[real].abs().clamp_min(1e-30)).max() if real.any() else 0.0) <= 2.0 ** -22


@pytest.mark.parametrize("metric", ["cosine", "euclidean"])
def test_metrics_at_the_ends(metric):
    B, T, dk = 2, 197, 192
    g = torch.Generator(device=DEV).manual_seed(3)
    q, k = (torch.randn(B, T, 1, dk, device=DEV, generator=g).bfloat16() for _ in range(2))
    n2 = [t.float().pow(2).sum(-1).permute(0, 2, 1).contiguous() for t in (q, k)]
    qs, ks = [t.rsqrt() for t in n2] if metric == "cosine" else n2
    spec = ops.LayerSpec(dk, 1, 9, "all", metric, "depthwise", True, False, T)
    idx, val = ops.sim_topk(spec, q, k, qs, ks)
    dot = torch.einsum("bthc,bshc->bhts", k.double(), q.double())
    if metric == "cosine":
        sim, sign = dot * ks.double().unsqueeze(-1) * qs.double().unsqueeze(2), 1.0
    else:
        sim, sign = (ks.double().unsqueeze(-1) + qs.double().unsqueeze(2) - 2 * dot).clamp_min(0).sqrt(), -1.0
    want = sign * (sign * sim).topk(9, -1).values
    # a dk-term fp32 sum of values whose squares add up to ~dk, relative to the distance / to 1
    bound = (dk + 16) * 2.0 ** -24 * (1.0 if metric == "cosine" else 4.0 * math.sqrt(dk))
    assert float((val.double() - want).abs().max()) <= bound
    assert float((torch.gather(sim, -1, idx.long()) - val.double()).abs().max()) <= bound


# Batches at which a CTA of the warp-per-row kernel has several segments (whole sequences, ends, ranges across heads), and
# some beside them that go to the two-pass and the streaming kernel (test_warp_per_row_routes has the lines).
@pytest.mark.parametrize("T,S,H,dk,K,B", [(197, 197, 1, 64, 9, 90), (197, 197, 3, 32, 9, 64), (197, 197, 1, 32, 9, 300),
                                          (150, 150, 1, 16, 16, 152), (1, 1, 1, 16, 1, 3000), (33, 17, 1, 32, 9, 150),
                                          (130, 130, 2, 64, 5, 74), (300, 200, 1, 48, 12, 149), (65, 65, 1, 64, 25, 60),
                                          (197, 64, 1, 64, 9, 74), (197, 197, 1, 64, 25, 60), (197, 64, 1, 64, 9, 200), (17, 17, 1, 32, 17, 278),
                                          (256, 256, 1, 64, 3, 55)])
@pytest.mark.parametrize("values", ["few", "many", "nan"])
def test_exact_lists_of_many_rows(T, S, H, dk, K, B, values):
    sampled = S != T
    n = K - 1 if sampled else K
    g = torch.Generator(device=DEV).manual_seed(T + S + K + B)
    top = 1 if values == "few" else 40               # products and sums stay below 2^24
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "nan":
        q[1::2, ::2] = math.nan
        q[2::3, 2:] = math.nan
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    idx, val = ops.sim_topk(spec, q.bfloat16(), k.bfloat16(), None, None, cand)
    key = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()        # whole numbers: exact
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV), key)
    want_idx, want_key = expect(key, n)
    want_tok = want_idx if cand is None else cand.long()[want_idx]
    assert torch.equal(idx.long()[..., K - n:], want_tok)
    if sampled:
        assert torch.equal(idx.long()[..., 0], torch.arange(T, device=DEV).expand(B, H, T))
    real = (want_key > -math.inf) & (want_tok != torch.arange(T, device=DEV).view(1, 1, T, 1) if sampled else want_key > -math.inf)
    want_val = want_key / torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV)
    # one division: equal up to its rounding
    assert bool(((val[..., K - n:] - want_val).abs()[real] <= 2.0 ** -22 * want_val.abs()[real]).all())


# float32 through the kernel that takes the whole candidate list at once: edges of its 32-row blocks, 32-column groups and
# 32-channel steps, and the last shape goes to the streaming kernel.
@pytest.mark.parametrize("T,S,H,dk,K,B", [(1, 1, 1, 3, 1, 1), (31, 31, 1, 32, 9, 2), (33, 33, 2, 33, 5, 2), (65, 65, 1, 192, 9, 3),
                                          (40, 32, 3, 20, 16, 2), (70, 64, 1, 31, 9, 2), (100, 97, 1, 64, 25, 2), (96, 96, 1, 65, 32, 2),
                                          (129, 129, 1, 16, 9, 2), (300, 150, 1, 48, 16, 2), (197, 197, 3, 64, 9, 4),
                                          (256, 256, 1, 7, 12, 2), (257, 225, 1, 40, 26, 2), (64, 40, 1, 8, 9, 500), (165, 165, 1, 33, 9, 2),
                                          (192, 192, 2, 16, 12, 2)])
@pytest.mark.parametrize("values", ["few", "many", "nan"])
def test_exact_lists_float32(T, S, H, dk, K, B, values):
    sampled = S != T
    n = K - 1 if sampled else K
    g = torch.Generator(device=DEV).manual_seed(T + S + K + dk)
    top = 1 if values == "few" else 50               # products and sums stay below 2^24
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "nan":
        q[:, ::3] = math.nan
        q[:1, 2:] = math.nan
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    idx, _ = ops.sim_topk(spec, q, k, None, None, cand)
    key = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()        # whole numbers: exact
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV), key)
    want_idx, _ = expect(key, n)
    assert torch.equal(idx.long()[..., K - n:], want_idx if cand is None else cand.long()[want_idx])


# Lines of the two rules: which kernel takes a batch just inside and just outside of each.
@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk,K,dtype,rows", [
    # bfloat16: at most 128 candidates and wide heads: 48 rows per SM, inside a head
    (139, 17, 17, 1, 384, 9, torch.bfloat16, True), (278, 17, 17, 1, 384, 9, torch.bfloat16, False), (109, 65, 40, 1, 768, 9, torch.bfloat16, False),
    (71, 100, 100, 1, 64, 9, torch.bfloat16, True), (74, 100, 100, 1, 64, 9, torch.bfloat16, False), (5, 197, 197, 1, 768, 9, torch.bfloat16, True),
    # more candidates, by the length of the list
    (37, 197, 197, 2, 32, 3, torch.bfloat16, True), (256, 130, 130, 1, 16, 3, torch.bfloat16, False), (192, 197, 197, 1, 192, 3, torch.bfloat16, False),
    (236, 130, 130, 1, 16, 5, torch.bfloat16, False), (140, 130, 130, 1, 16, 5, torch.bfloat16, True), (220, 197, 197, 1, 192, 9, torch.bfloat16, True),
    (256, 197, 197, 1, 192, 9, torch.bfloat16, False), (30, 1000, 250, 1, 384, 9, torch.bfloat16, False), (120, 256, 256, 1, 384, 9, torch.bfloat16, True),
    (64, 197, 197, 1, 192, 16, torch.bfloat16, True), (37, 1000, 250, 1, 192, 17, torch.bfloat16, False), (64, 197, 197, 1, 192, 13, torch.bfloat16, True),
    (16, 197, 197, 1, 192, 25, torch.bfloat16, True), (48, 197, 197, 1, 192, 25, torch.bfloat16, False),
    # float32: 8/3 CTAs per SM, then by the streaming kernel's work
    (32, 65, 65, 1, 192, 9, torch.float32, True), (64, 197, 197, 1, 192, 9, torch.float32, True), (150, 100, 100, 1, 192, 9, torch.float32, True),
    (230, 100, 100, 1, 192, 9, torch.float32, False), (18, 1000, 100, 1, 192, 9, torch.float32, False), (18, 1000, 100, 1, 16, 16, torch.float32, True),
    (75, 256, 256, 1, 400, 9, torch.float32, True), (115, 256, 256, 1, 400, 9, torch.float32, False), (152, 130, 130, 1, 400, 16, torch.float32, True),
    (230, 100, 100, 1, 16, 1, torch.float32, False), (109, 65, 40, 1, 16, 1, torch.float32, False), (64, 197, 64, 1, 384, 9, torch.float32, False),
    (300, 65, 65, 1, 192, 25, torch.float32, True), (131, 256, 256, 1, 33, 12, torch.float32, False)])
def test_warp_per_row_routes(B, T, S, H, dk, K, dtype, rows):
    g = torch.Generator(device=DEV).manual_seed(1)
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if S != T else "all", "matmul", "depthwise", True, False, T)
    q, k = (torch.randn(B, r, H, dk, device=DEV, generator=g).to(dtype) for r in (S, T))
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if S != T else None
    names = launches(lambda: ops.sim_topk(spec, q, k, None, None, cand))
    assert len(names) == 1 and any(n in next(iter(names)) for n in ("sim_topk_rows_kernel", "sim_topk_simt_rows_kernel")) == rows


@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk,K,two_pass", [
    # few candidates: narrow heads, several rounds of units, wide heads, long lists
    (1000, 17, 17, 1, 64, 5, True), (1000, 17, 17, 1, 512, 2, False), (340, 25, 25, 1, 192, 9, True), (200, 100, 20, 1, 384, 5, False),
    (340, 25, 25, 1, 768, 5, True), (281, 48, 33, 1, 128, 5, True), (281, 48, 33, 3, 64, 12, False), (512, 197, 16, 1, 192, 4, False),
    (163, 65, 65, 1, 128, 12, False), (281, 65, 65, 1, 128, 12, True),
    # the widest heads, most candidates, streaming units that fill most of a round
    (141, 256, 256, 1, 768, 5, False), (100, 256, 256, 1, 768, 5, True), (200, 256, 256, 1, 768, 5, True), (141, 224, 224, 1, 768, 5, True)])
def test_two_pass_routes(B, T, S, H, dk, K, two_pass):
    g = torch.Generator(device=DEV).manual_seed(1)
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if S != T else "all", "matmul", "depthwise", True, False, T)
    q, k = (torch.randn(B, r, H, dk, device=DEV, generator=g).bfloat16() for r in (S, T))
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if S != T else None
    name, = launches(lambda: ops.sim_topk(spec, q, k, None, None, cand))
    assert ("sim_topk_short_kernel" in name) == two_pass and ("sim_topk_tc_kernel" in name) != two_pass


# Several 128-row units per SM.  (80 x 197 x 64 with one accumulator in four and one in two; 33 to 48 candidates leave the upper
# half of a row a chunk or nothing; 208 and 256 end on a whole chunk; "few" values tie, so that most rows overflow their entries;
# "stripes" puts the best sixteen columns into one group of maxima.)
@pytest.mark.parametrize("B,T,S,H,dk", [(160, 17, 17, 1, 64), (80, 197, 33, 1, 64), (80, 197, 64, 1, 384), (160, 128, 128, 1, 192),
                                        (60, 129, 48, 3, 16), (80, 197, 197, 1, 32), (60, 300, 208, 1, 512), (320, 256, 256, 1, 64)])
@pytest.mark.parametrize("K", [1, 3, 8, 9, 12])
@pytest.mark.parametrize("values", ["few", "many", "nan", "stripes"])
def test_exact_lists_of_many_units(B, T, S, H, dk, K, values):
    sampled = S != T
    n = K - 1 if sampled else K
    if n < 1:
        pytest.skip("the row itself is all of the list")
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + S + K)
    top = 1 if values == "few" else 11               # products and sums stay far below 2^24
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "nan":
        q[:, ::3] = math.nan
        q[1, 2:] = math.nan
    if values == "stripes":
        q[:, ::16] = q[:, ::16].abs() + 12
        k = k.abs()
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    idx, val = ops.sim_topk(spec, q.bfloat16(), k.bfloat16(), None, None, cand)
    key = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32), key)
    want_idx, want_key = expect(key, n)
    assert torch.equal(idx.long()[..., K - n:], want_idx if cand is None else cand.long()[want_idx])
    real = (want_key > -math.inf) & ~((want_key < 0) & (val[..., K - n:] == -0.1))
    want_val = want_key / torch.tensor(math.sqrt(dk), dtype=torch.float32)
    # one division: equal up to its rounding
    assert bool(((val[..., K - n:] - want_val).abs() <= 2.0 ** -22 * want_val.abs())[real].all())


# The same kernel for the other metrics, whose rows end on a NaN statistic instead of -inf: whole numbers with statistics that are
# powers of two (cosine) or exact squared norms (euclidean), so that every key is exact.
@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk", [(160, 17, 17, 1, 64), (80, 197, 33, 1, 64), (80, 197, 64, 1, 384), (160, 128, 128, 1, 192),
                                        (60, 129, 48, 3, 16), (80, 197, 197, 3, 32), (60, 300, 208, 1, 512), (320, 256, 256, 1, 64)])
@pytest.mark.parametrize("K", [3, 9, 12])
@pytest.mark.parametrize("values", ["few", "many", "nan", "stripes"])
@pytest.mark.parametrize("metric", ["cosine", "euclidean"])
def test_exact_lists_of_the_other_metrics(B, T, S, H, dk, K, values, metric):
    sampled = S != T
    n = K - 1 if sampled else K
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + S + K)
    top = 1 if values == "few" else 11               # products and sums stay far below 2^24
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "stripes":
        q[:, ::16] = q[:, ::16].abs() + 12
        k = k.abs()
    if metric == "cosine":
        qs, ks = (2.0 ** torch.randint(-2, 3, (B, H, r), device=DEV, generator=g).float() for r in (S, T))
    else:
        qs, ks = (t.pow(2).sum(-1).permute(0, 2, 1).contiguous() for t in (q, k))
    if values == "nan":
        q[:, ::3] = math.nan
        q[1, 2:] = math.nan
        qs[:, :, 1::5] = math.nan
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", metric, "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    call = lambda: ops.sim_topk(spec, q.bfloat16(), k.bfloat16(), qs, ks, cand)
    if S > 40 or n <= 9:
        assert any("sim_topk_short_kernel" in name for name in launches(call))
    idx, val = call()
    dot = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()
    col, row = qs.unsqueeze(2), ks.unsqueeze(3)
    key = dot * col if metric == "cosine" else 2 * dot - col
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.tensor(-0.1, device=DEV) / row if metric == "cosine" else row - torch.tensor(1.21, device=DEV), key)
    want_idx, want_key = expect(key, n)
    token = want_idx if cand is None else cand.long()[want_idx]
    assert torch.equal(idx.long()[..., K - n:], token)
    want = want_key * row if metric == "cosine" else (row - want_key).clamp_min(0).sqrt()
    if sampled:
        self = token == torch.arange(T, device=DEV).view(1, 1, T, 1)
        want = torch.where(self, torch.tensor(-0.1 if metric == "cosine" else 1.1, device=DEV), want)
    real = want_key > -math.inf
    # one product, or a difference of whole numbers and its root: equal up to the root's rounding
    assert bool(((val[..., K - n:] - want).abs() <= 2.0 ** -22 * want.abs())[real].all())


# Lists of more than twelve, ranked by one thread per row, with several units per SM, and short ones written by lines (K = 9, 384 rows
# per SM, ragged ends).  "close" keys agree in all but their last bits, so that neighbours in the list and at its end are told
# apart by what the entries hold; "few" values tie and overflow the entries; "stripes" puts the best columns into few groups of maxima.
@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk", [(160, 40, 40, 1, 64), (100, 197, 64, 1, 384), (160, 128, 128, 1, 192), (60, 129, 48, 3, 16),
                                        (80, 197, 197, 3, 32), (60, 300, 208, 1, 512), (160, 256, 256, 1, 64), (325, 197, 197, 1, 32)])
@pytest.mark.parametrize("K", [9, 13, 16, 17, 25, 32])
@pytest.mark.parametrize("values", ["few", "many", "nan", "stripes", "close", "inf"])
def test_ranked_entries(B, T, S, H, dk, K, values):
    sampled = S != T
    n = K - 1 if sampled else K
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + S + K)
    top = 1 if values == "few" else 11               # products and sums stay below 2^24
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "nan":
        q[:, ::3] = math.nan
        q[1, 2:] = math.nan
    if values == "stripes":
        q[:, ::16] = q[:, ::16].abs() + 12
        k = k.abs()
    if values == "close":
        q[..., 0], k[..., 0] = 2048.0, 2048.0
    if values == "inf":
        q[:, 5], k[..., 0] = 1.0, 3.0
        q[:, 5, :, 0] = math.inf
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    idx, val = ops.sim_topk(spec, q.bfloat16(), k.bfloat16(), None, None, cand)
    key = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV), key)
    want_idx, want_key = expect(key, n)
    assert torch.equal(idx.long()[..., K - n:], want_idx if cand is None else cand.long()[want_idx])
    real = (want_key.abs() < math.inf) & ~((want_key < 0) & (val[..., K - n:] == -0.1))
    want_val = want_key / torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV)
    # one division: equal up to its rounding
    assert bool(((val[..., K - n:] - want_val).abs() <= 2.0 ** -22 * want_val.abs())[real].all())


# Lists of more than twelve whose first bound more columns reach than a row has entries: the best columns lie in few groups of maxima
# ("few groups"), the good ones come last ("rising"), so that the tighter bound is no help either, or first ("falling"), or tie there ("steps").
@on_148_sms
@pytest.mark.parametrize("B,T,S,dk", [(60, 256, 256, 64), (60, 300, 241, 96), (100, 128, 128, 64), (200, 65, 65, 32), (70, 255, 255, 384)])
@pytest.mark.parametrize("K", [13, 16, 17, 25, 31, 32])
@pytest.mark.parametrize("values", ["few groups", "rising", "falling", "steps", "nan", "inf"])
def test_more_columns_at_the_bound_than_entries(B, T, S, dk, K, values):
    sampled = S != T
    n = K - 1 if sampled else K
    g = torch.Generator(device=DEV).manual_seed(T * 1000 + S + K)
    q, k = (torch.randint(-2, 3, (B, r, 1, dk), device=DEV, generator=g).float() for r in (S, T))
    c = torch.arange(S, device=DEV)
    worth = {"rising": c, "falling": S - c, "steps": c // 8 * 8}.get(values, torch.randperm(S, device=DEV, generator=g))
    if values not in ("rising", "falling", "steps"):
        worth = worth + 256 * (c % 64 < 16)
    q[..., 0], k[..., 0] = (worth // 16).float().view(1, S, 1), 256.0     # 16 worth, and noise of up to 4 per other channel
    q[..., 1], k[..., 1] = (worth % 16).float().view(1, S, 1), 16.0
    if values == "nan":
        q[:, ::5] = math.nan
    if values == "inf":
        q[::2, 7, :, 2], k[..., 2] = math.inf, 1.0
    spec = ops.LayerSpec(dk, 1, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    call = lambda: ops.sim_topk(spec, q.bfloat16(), k.bfloat16(), None, None, cand)
    assert any("sim_topk_short_kernel" in name for name in launches(call))
    idx, val = call()
    key = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV), key)
    want_idx, want_key = expect(key, n)
    assert torch.equal(idx.long()[..., K - n:], want_idx if cand is None else cand.long()[want_idx])
    real = (want_key.abs() < math.inf) & ~((want_key < 0) & (val[..., K - n:] == -0.1))
    want_val = want_key / torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV)
    # one division: equal up to its rounding
    assert bool(((val[..., K - n:] - want_val).abs() <= 2.0 ** -22 * want_val.abs())[real].all())


# Lines between the two-pass and the warp-per-row kernel: either side of each.
@on_148_sms
@pytest.mark.parametrize("B,T,S,dk,K,rows", [
    (13, 900, 250, 64, 9, True), (20, 900, 250, 64, 9, False), (18, 900, 190, 32, 6, True), (20, 900, 190, 32, 6, False),
    (13, 860, 190, 256, 9, True), (16, 860, 190, 256, 9, False)])
def test_warp_per_row_or_two_passes(B, T, S, dk, K, rows):
    test_warp_per_row_routes(B, T, S, 1, dk, K, torch.bfloat16, rows)


# The same for long lists among few candidates, with the streaming kernel where it takes half the rounds.
@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk,K,kernel", [
    (27, 281, 30, 1, 64, 24, "rows"), (29, 385, 64, 1, 64, 18, "rows"), (37, 385, 64, 1, 64, 18, "short"),
    (50, 40, 20, 6, 32, 18, "rows"), (50, 41, 20, 6, 32, 18, "short"), (50, 50, 50, 6, 512, 30, "rows"), (50, 50, 50, 6, 496, 30, "short"),
    (148, 172, 40, 1, 32, 28, "tc"), (149, 172, 40, 1, 32, 28, "short"), (148, 172, 41, 1, 32, 28, "short"), (135, 132, 28, 2, 16, 28, "tc"),
    (300, 140, 28, 1, 16, 28, "tc"), (300, 161, 28, 1, 16, 28, "short"), (148, 172, 40, 1, 32, 18, "tc"), (135, 172, 31, 2, 16, 18, "short"), (32, 574, 18, 3, 512, 18, "tc"), (94, 153, 23, 1, 768, 17, "short")])
def test_long_lists_among_few_candidates(B, T, S, H, dk, K, kernel):
    g = torch.Generator(device=DEV).manual_seed(T + S + K)
    sampled, n = S != T, K - (S != T)
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    q, k = (torch.randint(-11, 12, (B, r, H, dk), device=DEV, generator=g).bfloat16() for r in (S, T))
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    call = lambda: ops.sim_topk(spec, q, k, None, None, cand)
    name, = launches(call)
    assert f"sim_topk_{kernel}_kernel" in name
    key = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()        # whole numbers: exact
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        key = torch.where(own, torch.full_like(key, -0.1) * torch.tensor(math.sqrt(dk), dtype=torch.float32, device=DEV), key)
    want_idx, _ = expect(key, n)
    assert torch.equal(call()[0].long()[..., K - n:], want_idx if cand is None else cand.long()[want_idx])
