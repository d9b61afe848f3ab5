"""The fp32-pipe kernels at the edges of their tiles: plain, three-output, neighbour and Conv1d operands of the SIMT
GEMM, and the register-blocked similarity / top-K kernel."""
import re

import pytest
import torch

from convnn_b200 import ops
from gpu_util import DEV, launches, on_148_sms

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


def _bound(a, w, terms):
    """|computed - exact| of a sum of `terms` fp32 products in any order: terms * eps * sum |a||w| (first order)."""
    return (terms + 2) * EPS * (a.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (31, 33, 15), (32, 64, 16), (65, 63, 17), (128, 128, 32), (129, 257, 100),
                                   (3000, 192, 192), (4097, 130, 36), (20000, 768, 20)])
def test_linear_float32(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N)
    a = torch.randn(M, K, device=DEV, generator=g)
    w = torch.randn(N, K, device=DEV, generator=g)
    b = torch.randn(N, device=DEV, generator=g)
    r = torch.randn(M, N, device=DEV, generator=g)
    got = ops.linear(a, w, b, residual=r)
    want = a.double() @ w.double().T + b.double() + r.double()
    err = (got.double() - want).abs()
    assert bool((err <= _bound(a, w, K) + 4 * EPS * (b.abs() + r.abs() + want.abs())).all())


@pytest.mark.parametrize("H,dk,T,coord", [(1, 20, 70, True), (3, 12, 197, False), (1, 193, 130, True), (1, 132, 257, False)])
@pytest.mark.parametrize("conv", ["standard", "depthwise-separable"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_matrix_convs_against_float64(H, dk, T, coord, conv, dtype):
    if conv == "standard" and dk % 4 and not coord:
        pytest.skip("stored widths that are no multiple of four take another kernel")
    B, K = 2, 5
    g = torch.Generator(device=DEV).manual_seed(dk + T)
    spec = ops.LayerSpec(H * dk, H, K, "all", "cosine", conv, True, coord, T)
    C = dk + int(coord)
    Cp = (C + 7) // 8 * 8 if coord else dk
    v = torch.zeros(B, T, H, Cp, device=DEV)
    v[..., :C] = torch.randn(B, T, H, C, device=DEV, generator=g)
    v = v.to(dtype)
    idx = torch.randint(0, T, (B, H, T, K), device=DEV, generator=g, dtype=torch.int32)
    val = torch.randn(B, H, T, K, device=DEV, generator=g)
    p = torch.softmax(val.double(), -1)
    rows = v.double().permute(0, 2, 1, 3)[..., :C]                        # (B, H, T, C)
    nb = torch.gather(rows.unsqueeze(3).expand(B, H, T, K, C), 2, idx.long().unsqueeze(-1).expand(B, H, T, K, C))
    nb = nb * p.unsqueeze(-1)
    if conv == "standard":
        w = (torch.randn(dk, K, C, device=DEV, generator=g) / (K * C) ** 0.5).to(dtype)
        got = ops.gather_conv(spec, v, idx, val, w)
        want = torch.einsum("bhtjc,ojc->bhto", nb, w.double())
        mass = torch.einsum("bhtjc,ojc->bhto", nb.abs(), w.double().abs())
        terms = K * C
    else:
        w = torch.randn(K, C, device=DEV, generator=g).to(dtype)
        pw = (torch.randn(dk, C, device=DEV, generator=g) / C ** 0.5).to(dtype)
        got = ops.gather_conv(spec, v, idx, val, w, pw)
        mid = torch.einsum("bhtjc,jc->bhtc", nb, w.double())
        want = torch.einsum("bhtc,oc->bhto", mid, pw.double())
        mass = torch.einsum("bhtc,oc->bhto", torch.einsum("bhtjc,jc->bhtc", nb.abs(), w.double().abs()), pw.double().abs())
        terms = K + C
    # fp32 sums (and softmax weights within a few eps) plus, in bfloat16, one rounding of the result; without the
    # coordinate channel the tensor-core route also rounds its operand once
    rel = (terms + 16) * EPS + (0 if dtype == torch.float32 else 2.0 ** -9 * (1 if coord else 2))
    assert bool(((got.double() - want).abs() <= rel * mass + (0 if dtype == torch.float32 else 2.0 ** -8) * want.abs() + 1e-30).all())


@pytest.mark.parametrize("ks", [1, 4, 9])
@pytest.mark.parametrize("T,dk", [(3, 4), (65, 12), (130, 36)])
def test_conv1d_branch_float32(T, dk, ks):
    g = torch.Generator(device=DEV).manual_seed(T)
    B, H, D = 2, 2, 2 * dk
    eye, zero = torch.eye(D, device=DEV), torch.zeros(D, device=DEV)
    x = torch.randn(B, T, D, device=DEV, generator=g)
    w = torch.randn(dk, ks, dk, device=DEV, generator=g)
    b = torch.randn(dk, device=DEV, generator=g)
    got = ops.conv1d_attention(x, eye, zero, w, b, eye, zero, H, ks)
    y = x.double().view(B, T, H, dk).permute(0, 2, 3, 1).reshape(B * H, dk, T)
    left = (ks - 1) // 2
    z = torch.nn.functional.conv1d(torch.nn.functional.pad(y, (left, ks - 1 - left)), w.double().permute(0, 2, 1), b.double())
    flat = z.permute(0, 2, 1).reshape(B, H, T * dk)                       # (t, c) rows read back as (c, t)
    want = flat.view(B, H, dk, T).permute(0, 3, 1, 2).reshape(B, T, D)
    scale = float(w.abs().sum(dim=(1, 2)).max()) * float(x.abs().max()) + float(b.abs().max())
    assert float((got.double() - want).abs().max()) <= (ks * dk + D + 4) * EPS * scale


# Every tile of the implicit operands in both its forms (outputs per thread), at the rounds of tiles per SM where the rule
# changes its mind; standard conv (coord: one channel more, in bfloat16), then the shifted rows of the Conv1d branch.
@on_148_sms
@pytest.mark.parametrize("B,T,H,dk,K,coord,tile", [
    (32, 197, 3, 64, 9, False, "128x64 8x4"), (256, 65, 1, 192, 9, False, "128x64 8x8"), (128, 197, 3, 64, 9, False, "128x64 8x4"),
    (8, 197, 1, 192, 9, False, "64x64 4x4"), (20, 577, 1, 100, 9, False, "64x64 8x4"), (64, 197, 1, 192, 9, False, "64x64 4x4"),
    (32, 197, 1, 384, 2, False, "64x64 8x4"), (8, 197, 3, 64, 9, False, "32x64 4x2"), (1, 197, 3, 64, 9, False, "32x32 4x2"),
    (64, 197, 2, 20, 9, False, "32x32 4x4"), (16, 197, 1, 192, 9, True, "128x64 8x4"), (24, 577, 1, 96, 16, True, "64x64 8x4"),
    (64, 197, 1, 192, 5, True, "64x64 4x4"), (24, 577, 1, 96, 8, True, "64x64 8x4"), (24, 197, 1, 384, 3, True, "64x64 4x4"),
    (159, 65, 1, 96, 25, True, "32x32 4x2"), (48, 577, 1, 20, 16, True, "32x32 4x4")])
def test_standard_conv_tiles_of_the_simt_gemm(B, T, H, dk, K, coord, tile):
    dtype = torch.bfloat16 if coord else torch.float32
    C = dk + int(coord)
    Cp = (C + 7) // 8 * 8 if coord else dk
    g = torch.Generator(device=DEV).manual_seed(B + T + dk)
    spec = ops.LayerSpec(H * dk, H, K, "all", "cosine", "standard", True, coord, T)
    v = torch.zeros(B, T, H, Cp, device=DEV)
    v[..., :C] = torch.randn(B, T, H, C, device=DEV, generator=g)
    v = v.to(dtype)
    idx = torch.randint(0, T, (B, H, T, K), device=DEV, generator=g, dtype=torch.int32)
    val = torch.randn(B, H, T, K, device=DEV, generator=g)
    w = (torch.randn(dk, K, C, device=DEV, generator=g) / (K * C) ** 0.5).to(dtype)
    assert _tiles(lambda: ops.gather_conv(spec, v, idx, val, w)) == {tile}
    got = ops.gather_conv(spec, v, idx, val, w)
    p = torch.softmax(val.double(), -1)
    rows = v.double().permute(0, 2, 1, 3)[..., :C]
    want, mass = torch.zeros(B, H, T, dk, device=DEV, dtype=torch.double), torch.zeros(B, H, T, dk, device=DEV, dtype=torch.double)
    for j in range(K):
        nb = p[..., j:j + 1] * torch.gather(rows, 2, idx[..., j:j + 1].long().expand(B, H, T, C))
        want += nb @ w[:, j].double().T
        mass += nb.abs() @ w[:, j].double().abs().T
    # fp32 sums of K * C terms, softmax weights within a few eps; in bfloat16 one rounding of the result
    bound = (K * C + 16) * EPS * mass + (2.0 ** -8 * want.abs() if coord else 0) + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())


def _tiles(fn):
    names = [re.search(r"gemm_simt_kernelI.*?Li[34]ELi(\d+)ELi(\d+)ELi\d+ELi(\d+)ELi(\d+)E", n) for n in launches(fn)]
    return {"{}x{} {}x{}".format(*m.groups()) for m in names if m}


@on_148_sms
@pytest.mark.parametrize("B,T,H,dk,ks,tile", [(16, 197, 1, 192, 9, "128x64 8x4"), (64, 197, 1, 192, 3, "64x64 8x4"),
                                              (8, 197, 1, 192, 4, "64x64 4x4"), (32, 197, 1, 192, 3, "32x64 4x4"),
                                              (8, 197, 1, 96, 9, "32x64 4x2"), (1, 197, 3, 32, 9, "32x32 4x2"), (64, 197, 2, 20, 9, "32x32 4x4")])
def test_conv1d_tiles_of_the_simt_gemm(B, T, H, dk, ks, tile):
    D = H * dk
    g = torch.Generator(device=DEV).manual_seed(B + T + dk)
    eye, zero = torch.eye(D, device=DEV), torch.zeros(D, device=DEV)
    x = torch.randn(B, T, D, device=DEV, generator=g)
    w = torch.randn(dk, ks, dk, device=DEV, generator=g)
    b = torch.randn(dk, device=DEV, generator=g)
    call = lambda: ops.conv1d_attention(x, eye, zero, w, b, eye, zero, H, ks)
    assert _tiles(call) == {tile}
    left = (ks - 1) // 2
    y = torch.nn.functional.pad(x.double().view(B, T, H, dk).permute(0, 2, 1, 3), (0, 0, left, ks - 1 - left))
    z = b.double().expand(B, H, T, dk).clone()
    mass = b.double().abs().expand(B, H, T, dk).clone()
    for j in range(ks):
        z += y[:, :, j:j + T] @ w[:, j].double().T
        mass += y[:, :, j:j + T].abs() @ w[:, j].double().abs().T
    flat = lambda t: t.reshape(B, H, dk, T).permute(0, 3, 1, 2).reshape(B, T, D)       # (t, c) rows read back as (c, t)
    # fp32 sums of ks * dk terms between two products with the identity
    assert bool(((call().double() - flat(z)).abs() <= (ks * dk + 8) * EPS * flat(mass) + 1e-30).all())


@pytest.mark.parametrize("T,S,C,K", [(1, 1, 4, 1), (63, 64, 20, 9), (65, 65, 16, 25), (129, 200, 33, 32), (257, 63, 48, 4),
                                     (300, 300, 8, 16), (2500, 65, 36, 9), (65, 65, 24, 8), (130, 130, 20, 12),
                                     (197, 70, 36, 11)])
@pytest.mark.parametrize("metric", ["cosine", "matmul", "euclidean"])
def test_similarity_lists_float32(T, S, C, K, metric):
    g = torch.Generator(device=DEV).manual_seed(T + S)
    B = 2 if T < 2000 else 8
    spec = ops.LayerSpec(C, 1, K, "random", metric, "depthwise", True, False, T) if S != T else \
        ops.LayerSpec(C, 1, K, "all", metric, "depthwise", True, False, T)
    cand = torch.randint(0, T, (S,), device=DEV, generator=g, dtype=torch.int32) if S != T else None
    q = torch.randn(B, S, 1, C, device=DEV, generator=g)
    k = torch.randn(B, T, 1, C, device=DEV, generator=g)
    q[:, S // 2] = q[:, 0]                                                # an exact tie: the lower column goes first
    qs, ks = q.double().square().sum(-1).view(B, 1, S), k.double().square().sum(-1).view(B, 1, T)
    if metric == "cosine":
        qs, ks = 1 / qs.sqrt(), 1 / ks.sqrt()
    idx, val = ops.sim_topk(spec, q, k, qs.float(), ks.float(), cand)
    sim = torch.einsum("btc,bsc->bts", k[:, :, 0].double(), q[:, :, 0].double())
    if metric == "cosine":
        sim = sim * ks.view(B, T, 1) * qs.view(B, 1, S)
    elif metric == "matmul":
        sim = sim / C ** 0.5
    else:
        sim = -(ks.view(B, T, 1) + qs.view(B, 1, S) - 2 * sim).clamp_min(0).sqrt()
    if cand is not None:
        own = cand.view(1, 1, S).long() == torch.arange(T, device=DEV).view(1, T, 1)
        sim = sim.masked_fill(own, -1.1 if metric == "euclidean" else -0.1)
    n = K if cand is None else K - 1
    if n == 0:
        return
    sign = -1 if metric == "euclidean" else 1
    want = sim.topk(n, -1).values
    got, chosen = idx[:, 0, :, K - n:].long(), val[:, 0, :, K - n:].double() * sign
    # rounding of a C-term fp32 dot product and of the few operations behind it, for the largest products of the row; a
    # distance is the root of a difference: its error is that of the difference over the distance, its root near zero
    kn, qn = k[:, :, 0].double().norm(dim=-1, keepdim=True), q[:, :, 0].double().norm(dim=-1).amax(-1).view(B, 1, 1)
    if metric == "cosine":
        tol = torch.full_like(kn, (C + 16) * EPS)
    elif metric == "matmul":
        tol = (C + 16) * EPS * kn * qn / C ** 0.5
    else:
        square = (C + 16) * EPS * (kn + qn) ** 2
        tol = torch.minimum(square.sqrt(), square / want.abs().clamp_min(1e-30))
    assert bool(((chosen - want).abs() <= tol).all())
    # ... and is the value of the token it is reported for (candidates may hold a token several times)
    column = torch.arange(S, device=DEV) if cand is None else cand.long()
    near = torch.where(column.view(1, 1, 1, S) == got.unsqueeze(-1), (sim.unsqueeze(2) - chosen.unsqueeze(-1)).abs(),
                       torch.full((), float("inf"), device=DEV, dtype=torch.float64)).amin(-1)
    assert bool((near <= tol).all())
    if cand is None:
        assert all(len(set(r.tolist())) == n for r in got.view(-1, n)[:200])
        first = (got == 0).int().argmax(-1)
        tied = (got == S // 2).int().argmax(-1)
        both = (got == 0).any(-1) & (got == S // 2).any(-1)
        assert S < 2 or bool((first[both] < tied[both]).all())


@pytest.mark.parametrize("B,T,S,H,dk,coord,dtype", [(3, 65, 65, 2, 16, False, torch.bfloat16), (2, 100, 40, 1, 20, True, torch.bfloat16),
                                                    (2, 50, 50, 3, 12, False, torch.float32), (1, 33, 20, 1, 24, True, torch.float32)])
@pytest.mark.parametrize("metric", ["cosine", "euclidean"])
def test_statistics_of_all_tensors_in_one_launch(B, T, S, H, dk, coord, dtype, metric):
    """Norms of the stored q and k, the coordinate channel of all three, and a kernel without local memory."""
    D, C = H * dk, dk + int(coord)
    g = torch.Generator(device=DEV).manual_seed(T)
    spec = ops.LayerSpec(D, H, 5, "spatial" if S != T else "all", metric, "standard", True, coord, T)
    x, w = (torch.randn(*s, device=DEV, generator=g).to(dtype) for s in ((B, T, D), (3, D, D)))
    cand = torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32) if S != T else None
    names = {n: local for n, local in launches(lambda: ops.qkv_proj(spec, x, w, cand)).items() if "head_stats_kernel" in n}
    assert list(names.values()) == [0]
    q, k, v, qs, ks = ops.qkv_proj(spec, x, w, cand)
    for t, stat, rows in ((q, qs, S), (k, ks, T), (v, None, T)):
        if coord:
            ramp = torch.linspace(-1, 1, rows, device=DEV).to(dtype).view(1, rows, 1)
            assert bool(((t[..., dk] - ramp).abs() <= 2.0 ** -8).all()) and not bool(t[..., C:].any())
        if stat is None:
            continue
        want = t[..., :C].double().square().sum(-1).permute(0, 2, 1)
        want = 1 / want.sqrt().clamp_min(1e-12) if metric == "cosine" else want
        # a C-term fp32 sum of squares, a root and a division
        assert bool(((stat.view(B, H, rows).double() - want).abs() <= (C + 8) * EPS * want.abs() + 1e-30).all())


# Every tile of the float32 rows (columns of a tile x outputs per thread; "transposed": those that are), with ragged rows,
# columns and k; a sum is the same whichever tile it was computed in.
@on_148_sms
@pytest.mark.parametrize("M,N,K,tile", [
    (2081, 190, 100, "32x32 4x4"), (1, 1, 4, "transposed"), (1, 1, 132, "32x32 4x4"), (33, 65, 768, "32x32 4x4"), (3121, 190, 764, "32x32 4x4"),
    (5003, 193, 36, "transposed"), (1576, 385, 100, "40x32 5x4"), (1001, 1003, 192, "40x32 5x4"), (500, 64, 96, "transposed"),
    (5003, 192, 36, "40x32 5x4"), (1301, 64, 96, "transposed"), (3200, 64, 96, "32x32 4x4"), (5003, 192, 20, "transposed"), (2081, 190, 768, "48x32 6x4"),
    (1050, 383, 388, "48x32 6x4"), (5203, 190, 768, "56x32 7x4"), (2081, 577, 32, "transposed"), (50432, 190, 8, "transposed")])
def test_tiles_of_float32_rows(M, N, K, tile):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a, w, b, r = (torch.randn(*s, device=DEV, generator=g) for s in ((M, K + 4), (N, K), (N,), (M, N)))
    a = a[:, :K]                                                     # rows K + 4 values apart
    call = lambda: ops.linear(a, w, b, residual=r)
    names = [re.search(r"gemm_simt_copy_kernelILi\dELi(\d+)ELi(\d+)ELi(\d+)ELi(\d+)E", n) for n in launches(call)]
    assert [("{}x{} {}x{}".format(*m.groups()) if m else "transposed") for m in names] == [tile]
    got = call()
    want = a.double() @ w.double().T + b.double() + r.double()
    assert bool(((got.double() - want).abs() <= _bound(a, w, K) + 4 * EPS * (b.abs() + r.abs() + want.abs())).all())
    some = torch.randperm(M, device=DEV, generator=g)[:20]
    assert torch.equal(ops.linear(a[some], w, b, residual=r[some]), got[some])


@pytest.mark.parametrize("B,T,S,D,H", [(8, 197, 49, 192, 3), (2, 50, 50, 96, 1), (33, 65, 65, 192, 1)])
def test_three_outputs_of_float32_rows(B, T, S, D, H):
    g = torch.Generator(device=DEV).manual_seed(T)
    spec = ops.LayerSpec(D, H, 9, "all" if S == T else "spatial", "matmul", "depthwise", True, False, T)
    x, w = torch.randn(B, T, D, device=DEV, generator=g), torch.randn(3, D, D, device=DEV, generator=g)
    cand = None if S == T else torch.randperm(T, device=DEV, generator=g)[:S].to(torch.int32)
    q, k, v = ops.qkv_proj(spec, x, w, cand)[:3]
    xq = x if cand is None else x[:, cand.long()]
    for got, rows, part in ((k, x, 0), (v, x, 1), (q, xq, 2)):
        assert torch.equal(got.reshape(-1, D), ops.linear(rows.reshape(-1, D), w[part]))


# Every tile of the rows that are not copied: bfloat16 with k a multiple of four (read four at a time) and not, and float32 rows
# that are not 16-byte aligned ("staged" through registers, or transposed); a sum is the same whichever tile it was computed in.
@on_148_sms
@pytest.mark.parametrize("M,N,K,bf16,fp32", [
    (1, 1, 1, "32x32", "32x32"), (65, 193, 385, "32x64 staged", "32x32"), (1050, 384, 388, "32x64 staged", "64x64"),
    (788, 768, 772, "40x32 staged", "32x64 staged"), (1576, 191, 196, "40x32 staged", "32x32"), (4039, 384, 385, "64x64 staged", "64x64"),
    (12001, 384, 197, "64x64 staged", "128x64"), (50433, 66, 65, "64x64 staged", "128x64"), (50433, 66, 68, "128x64", "128x64"),
    (12001, 16, 17, "32x32", "32x32"), (5001, 24, 28, "32x32", "32x32")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tiles_of_staged_rows(M, N, K, bf16, fp32, dtype):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    ld = K + (1 if dtype == torch.float32 or K % 4 else 4)           # (odd row strides keep float32 off the copies)
    a, w, b, r = (torch.randn(*s, device=DEV, generator=g).to(dtype) for s in ((M, ld), (N, K), (N,), (M, N)))
    a = a[:, :K]
    call = lambda: ops.linear(a, w, b, residual=r)
    names = [re.search(r"gemm_simt_(stage_|copy_|)kernelI.*?Li\dELi(\d+)ELi(\d+)E", n).groups() for n in launches(call)]
    assert [f"{bm}x{bn}" + {"stage_": " staged", "copy_": " copied", "": ""}[kind] for kind, bm, bn in names] == \
        [fp32 if dtype == torch.float32 else bf16]
    got = call()
    want = a.double() @ w.double().T + b.double()
    step = 2.0 ** -8 if dtype == torch.bfloat16 else 2 * EPS         # the sum is rounded, then the skip connection added
    bound = _bound(a, w, K) + 2 * EPS * b.abs() + step * (want.abs() + (want + r.double()).abs())
    assert bool(((got.double() - want - r.double()).abs() <= bound).all())
    some = torch.randperm(M, device=DEV, generator=g)[:20]
    assert torch.equal(ops.linear(a[some], w, b, residual=r[some]), got[some])


# The 128 x 64 tile on bfloat16 and mixed rows, which stay as they came until they are stored to shared memory: ragged rows, columns
# and k, by fours and one by one (the separable conv's intermediate with the coordinate channel: dk + 1 values).
@on_148_sms
@pytest.mark.parametrize("B,T,dk", [(32, 197, 384), (25, 197, 768), (65, 577, 96), (48, 577, 96)])
def test_large_tile_of_mixed_rows(B, T, dk):
    g = torch.Generator(device=DEV).manual_seed(dk)
    spec = ops.LayerSpec(dk, 1, 5, "all", "cosine", "depthwise-separable", True, True, T)
    C, Cp = dk + 1, (dk + 8) // 8 * 8
    v = torch.zeros(B, T, 1, Cp, device=DEV)
    v[..., :C] = torch.randn(B, T, 1, C, device=DEV, generator=g)
    v = v.to(torch.bfloat16)
    idx = torch.randint(0, T, (B, 1, T, 5), device=DEV, generator=g, dtype=torch.int32)
    val = torch.randn(B, 1, T, 5, device=DEV, generator=g)
    dw = (torch.randn(5, C, device=DEV, generator=g) / 2).to(torch.bfloat16)
    pw = (torch.randn(dk, C, device=DEV, generator=g) / C ** 0.5).to(torch.bfloat16)
    call = lambda n=B: ops.gather_conv(spec, v[:n], idx[:n], val[:n], dw, pw)
    assert any(re.search(r"gemm_simt_kernelIf13__nv_bfloat16Li\dELi128ELi64E", n) for n in launches(call))
    got = call()
    assert torch.equal(call(2), got[:2])                             # (two images take smaller tiles: the same sums)


# The smallest tile on bfloat16 and mixed rows: its times are for eight of them on an SM.
@pytest.mark.parametrize("M,N,K", [(37529, 32, 9), (4880, 192, 20)])
def test_eight_small_tiles_fit_an_sm(M, N, K):
    a, w = torch.ones(M, K, dtype=torch.bfloat16, device=DEV), torch.ones(N, K, dtype=torch.bfloat16, device=DEV)
    regs = {n: r for n, r in launches(lambda: ops.linear(a, w), "NUM_REGS").items() if "gemm_simt_kernel" in n}
    (name, r), = regs.items()
    assert "Li32ELi32ELi32ELi4ELi4E" in name and 8 * 64 * ((r + 7) // 8 * 8) <= 65536
    assert bool((ops.linear(a, w) == K).all())
