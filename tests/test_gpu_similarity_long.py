"""The pair kernel's selection under ties: small whole numbers, whose products and sums are exact, so that every list is known."""
import pytest
import torch

from convnn_b200 import ops
from gpu_util import DEV, launches, on_148_sms

pytestmark = pytest.mark.gpu


# Whole tiles of 256 columns and a ragged end; an upper half of the last tile that is padding; even and odd lists (the two
# halves' shares differ); rows that are all ties, and keys that grow or fall with the column, so that one half of a tile always
# sees the better ones first.
@pytest.mark.parametrize("T,S,dk,K", [(1100, 1100, 128, 9), (1024, 1024, 128, 5), (1030, 1153, 192, 16), (1281, 1040, 128, 12),
                                      (8192, 4096, 128, 25), (8200, 4225, 128, 26), (8192, 4100, 128, 32)])
@pytest.mark.parametrize("order", ["mixed", "rising", "falling"])
def test_ties_go_to_the_lower_column(T, S, dk, K, order):
    T = max(T, S)
    g = torch.Generator(device=DEV).manual_seed(T + S + K)
    spec = ops.LayerSpec(dk, 1, K, "all" if S == T else "spatial", "matmul", "depthwise", True, False, T)
    q = torch.randint(-1, 2, (1, S, 1, dk), device=DEV, generator=g).float()
    k = torch.randint(-1, 2, (1, T, 1, dk), device=DEV, generator=g).float()
    k[:, 5] = 0                                                # every key of this row is the same
    if order != "mixed":                                       # steps of 64 columns, more than the rest of a product reaches
        step = (torch.arange(S, device=DEV) // 64).float()
        q[0, :, 0, 0] = step if order == "rising" else step.flip(0)
        k[..., 0] = 4.0
        k[:, 5] = 0
    cand = None if S == T else torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32)
    qb, kb = q.bfloat16(), k.bfloat16()
    call = lambda: ops.sim_topk(spec, qb, kb, None, None, cand)
    assert any("sim_topk_tc2_kernel" in n for n in launches(call))
    idx, val = call()
    key = k[0, :, 0] @ q[0, :, 0].T                            # exact: whole numbers below 2^24
    n, first = K, 0
    if cand is not None:
        own = cand.view(1, S).long() == torch.arange(T, device=DEV).view(T, 1)
        key = key.masked_fill(own, -0.1 * dk ** 0.5)
        n, first = K - 1, 1
        assert torch.equal(idx[0, 0, :, 0].long(), torch.arange(T, device=DEV))
    col = key.sort(dim=1, descending=True, stable=True).indices[:, :n]
    want = col if cand is None else cand.long()[col]
    assert torch.equal(idx[0, 0, :, first:].long(), want)


# Columns that are no number, columns whose keys are +inf for some rows and -inf or no number for others, and rows with fewer
# usable columns than the list is long: NaN and -inf are never picked, an empty slot holds the first token.
@pytest.mark.parametrize("T,S,dk,K", [(1100, 1100, 128, 9), (1030, 1153, 192, 16), (2048, 2048, 64, 4), (8200, 4225, 128, 26)])
@pytest.mark.parametrize("columns", ["nan", "inf", "few left"])
def test_unusable_keys(T, S, dk, K, columns):
    T = max(T, S)
    g = torch.Generator(device=DEV).manual_seed(T + S + K)
    spec = ops.LayerSpec(dk, 1, K, "all" if S == T else "spatial", "matmul", "depthwise", True, False, T)
    q = torch.randint(-3, 4, (1, S, 1, dk), device=DEV, generator=g).float()
    k = torch.randint(-3, 4, (1, T, 1, dk), device=DEV, generator=g).float()
    if columns == "nan":
        q[:, ::3] = float("nan")
    elif columns == "inf":
        q[:, 7::50, :, 0] = float("inf")                       # times k's channel 0: both infinities, or no number at 0
        q[:, 100::200, :, 1] = float("-inf")
    else:
        q[:, 3:S - 2] = float("nan")
    cand = None if S == T else torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32)
    qb, kb = q.bfloat16(), k.bfloat16()
    call = lambda: ops.sim_topk(spec, qb, kb, None, None, cand)
    assert any("sim_topk_tc2_kernel" in name for name in launches(call))
    idx, val = call()
    dot = torch.zeros(T, S, device=DEV)
    for c in range(dk):                                        # (term by term: no infinity meets one that a sum made)
        dot += k[0, :, 0, c:c + 1] * q[0, :, 0, c]
    n, first = K, 0
    if cand is not None:
        own = cand.view(1, S).long() == torch.arange(T, device=DEV).view(T, 1)
        dot = dot.masked_fill(own, -0.1 * dk ** 0.5)
        n, first = K - 1, 1
    dot = torch.where(dot.isnan(), torch.full_like(dot, -float("inf")), dot)
    ranked = dot.sort(dim=1, descending=True, stable=True)
    col = torch.where(ranked.values[:, :n] > -float("inf"), ranked.indices[:, :n], 0)
    assert torch.equal(idx[0, 0, :, first:].long(), col if cand is None else cand.long()[col])


# Few units: two, four and eight CTAs per unit, some without a column tile, ragged last tiles, rows that end inside a CTA's share of the
# merge, lists longer than a CTA's share of good columns ("rising": all of the best lie in the last CTA's), ties and NaN.
@pytest.mark.parametrize("B,T,S,H,dk", [(1, 300, 300, 1, 64), (2, 577, 577, 1, 384), (1, 1040, 1040, 1, 256), (3, 1020, 344, 1, 512), (5, 700, 700, 2, 16),
                                        (1, 2600, 1100, 1, 256), (1, 2048, 2048, 1, 32)])
@pytest.mark.parametrize("K", [2, 5, 9, 12, 16, 25, 32])
@pytest.mark.parametrize("values", ["ties", "many", "rising", "nan"])
def test_columns_shared_by_a_cluster(B, T, S, H, dk, K, values, dtype=torch.bfloat16, kernel="sim_topk_tc_kernel"):
    g = torch.Generator(device=DEV).manual_seed(T + S + K)
    sampled = S != T
    top = 1 if values == "ties" else 11
    q, k = (torch.randint(-top, top + 1, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "rising":
        q[..., 0] = (torch.arange(S, device=DEV) // 8).float().view(1, S, 1)
        k[..., 0] = 16.0
    if values == "nan":
        q[:, ::3] = float("nan")
        q[0, 3:S - 2] = float("nan")
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", "matmul", "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    qb, kb = q.to(dtype), k.to(dtype)
    call = lambda: ops.sim_topk(spec, qb, kb, None, None, cand)
    assert any(kernel in name for name in launches(call))
    idx, val = call()
    key = torch.einsum("bthc,bshc->bhts", kb.double(), qb.double()).float()        # whole numbers below 2^24: exact
    n = K - 1 if sampled else K
    if sampled:
        own = cand.view(1, S).long() == torch.arange(T, device=DEV).view(T, 1)
        key = key.masked_fill(own, -0.1 * dk ** 0.5)
    key = torch.where(key.isnan(), torch.full_like(key, -float("inf")), key)
    ranked = key.sort(dim=-1, descending=True, stable=True)
    col = torch.where(ranked.values[..., :n] > -float("inf"), ranked.indices[..., :n], 0)
    assert torch.equal(idx.long()[..., K - n:], col if cand is None else cand.long()[col])


# The same on the fp32 pipes: blocks of 64 and of 128 rows, two to eight CTAs each, widths that are no multiple of four.
@pytest.mark.parametrize("B,T,S,H,dk", [(1, 300, 300, 1, 33), (2, 577, 577, 1, 64), (1, 1040, 1040, 1, 48), (1, 2100, 700, 1, 20), (2, 1300, 1300, 1, 64)])
@pytest.mark.parametrize("K", [4, 9, 16, 25, 32])
@pytest.mark.parametrize("values", ["ties", "many", "rising", "nan"])
def test_columns_shared_by_a_cluster_float32(B, T, S, H, dk, K, values):
    test_columns_shared_by_a_cluster(B, T, S, H, dk, K, values, torch.float32, "sim_topk_simt_kernel")


# 64 rows per CTA: the rule that shares columns counts on two CTAs per SM, also with the longest lists.
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("K", [4, 9, 16, 25, 32])
def test_two_blocks_of_64_rows_fit_an_sm(K, dtype):
    spec = ops.LayerSpec(97, 1, K, "all", "matmul", "depthwise", True, False, 439)
    q, k = (torch.ones(20, 439, 1, 97, device=DEV, dtype=dtype) for _ in "qk")
    regs = launches(lambda: ops.sim_topk(spec, q, k, None, None), "NUM_REGS")
    assert len(regs) == 1
    name, n = regs.popitem()
    assert "sim_topk_simt_kernel" in name and "Li64EEE" in name and 2 * 256 * ((n + 7) // 8 * 8) <= 65536


# Clusters that run at once: 15 of eight CTAs, 33 of four; beyond that fewer CTAs per unit, and a pair of SMs where it would be two.
@on_148_sms
@pytest.mark.parametrize("B,T,dk,K,kernel", [
    (1, 3840, 256, 9, "sim_topk_tc_kernel"), (1, 4096, 256, 16, "sim_topk_tc_kernel"), (3, 2816, 320, 12, "sim_topk_tc_kernel"), (3, 2816, 208, 12, "sim_topk_tc2_kernel"), (2, 4352, 256, 9, "sim_topk_tc2_kernel"),
    (2, 4352, 256, 16, "sim_topk_tc2_kernel"), (2, 4352, 256, 25, "sim_topk_tc_kernel")])
def test_clusters_that_run_at_once(B, T, dk, K, kernel):
    test_columns_shared_by_a_cluster(B, T, T, 1, dk, K, "many", kernel=kernel)


# What the merged lists are written as: values of the three metrics, the sampled rows' own entry, rows that pick themselves (every euclidean
# one, and the others where all products are negative), keys of +inf.  Whole numbers with statistics that are powers of two (cosine) or
# exact squared norms (euclidean), so that every key is exact.
@on_148_sms
@pytest.mark.parametrize("B,T,S,H,dk,dtype", [
    (1, 300, 300, 1, 64, torch.bfloat16), (3, 1020, 344, 1, 512, torch.bfloat16), (1, 2600, 1100, 1, 256, torch.bfloat16), (5, 700, 500, 2, 16, torch.bfloat16),
    (2, 577, 577, 1, 64, torch.float32), (1, 2100, 700, 1, 20, torch.float32), (1, 333, 270, 1, 33, torch.float32)])
@pytest.mark.parametrize("K", [4, 9, 13, 26])
@pytest.mark.parametrize("metric,values", [("cosine", "many"), ("cosine", "negative"), ("euclidean", "many"), ("matmul", "many"), ("matmul", "negative"),
                                           ("matmul", "inf")])
def test_values_of_lists_shared_by_a_cluster(B, T, S, H, dk, dtype, K, metric, values):
    g = torch.Generator(device=DEV).manual_seed(T + S + K)
    sampled, n = S != T, K - (S != T)
    q, k = (torch.randint(-11, 12, (B, r, H, dk), device=DEV, generator=g).float() for r in (S, T))
    if values == "negative":
        q, k = q.abs() + 1, -k.abs() - 1
    if values == "inf":
        q[:, 7::50, :, 2] = float("inf")
        k[..., 2] = torch.where(k[..., 2] < 0, -1.0, 1.0)
    qs, ks = (2.0 ** torch.randint(-2, 3, (B, H, r), device=DEV, generator=g).float() for r in (S, T))
    if metric == "euclidean":
        qs, ks = (t.pow(2).sum(-1).permute(0, 2, 1).contiguous() for t in (q, k))
    spec = ops.LayerSpec(H * dk, H, K, "spatial" if sampled else "all", metric, "depthwise", True, False, T)
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if sampled else None
    call = lambda: ops.sim_topk(spec, q.to(dtype), k.to(dtype), qs, ks, cand)
    kernel = "sim_topk_tc_kernel" if dtype == torch.bfloat16 else "sim_topk_simt_kernel"
    assert any(kernel in name for name in launches(call))
    idx, val = call()
    root = torch.tensor(dk, dtype=torch.float32, device=DEV).sqrt()
    dot = torch.einsum("bthc,bshc->bhts", k.double(), q.double()).float()
    col, row = qs.unsqueeze(2), ks.unsqueeze(3)
    key = {"cosine": dot * col, "euclidean": 2 * dot - col, "matmul": dot}[metric]
    if sampled:
        own = cand.view(1, 1, 1, S).long() == torch.arange(T, device=DEV).view(1, 1, T, 1)
        tenth = torch.tensor(-0.1, device=DEV)
        key = torch.where(own, {"cosine": tenth / row, "euclidean": row - torch.tensor(1.21, device=DEV), "matmul": tenth * root}[metric], key)
    ranked = torch.where(key.isnan(), -float("inf"), key).sort(dim=-1, descending=True, stable=True)
    want_key = ranked.values[..., :n]
    want_idx = torch.where(want_key > -float("inf"), ranked.indices[..., :n], 0)
    token = want_idx if cand is None else cand.long()[want_idx]
    assert torch.equal(idx.long()[..., K - n:], token)
    want = {"cosine": want_key * row, "euclidean": (row - want_key).clamp_min(0).sqrt(), "matmul": want_key / root}[metric]
    if sampled:
        here = torch.arange(T, device=DEV).view(1, 1, T, 1)
        want = torch.where(token == here, torch.tensor(1.1 if metric == "euclidean" else -0.1, device=DEV), want)
        assert torch.equal(idx.long()[..., :1], here.expand(B, H, T, 1)) and bool((val[..., 0] == 1).all())
        assert values != "negative" and metric != "euclidean" or bool((token == here).any())
    real = want_key.abs() < float("inf")
    # one product or quotient, or a difference of whole numbers and its root: equal up to that rounding
    assert bool(((val[..., K - n:] - want).abs() <= 2.0 ** -22 * want.abs())[real].all())
