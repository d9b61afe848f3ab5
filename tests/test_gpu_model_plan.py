"""The one-call ViT forward (host plan) against the op-by-op path: same kernels, so the same bits; and every change
of the model that a plan must notice."""
import copy

import pytest
import torch

import convnn_b200
from convnn_b200 import model_plan

pytestmark = pytest.mark.gpu
DEV = "cuda"

CONFIGS = {
    "tiny": dict(layer="ConvNNAttention", num_heads=1, d_hidden=192, d_mlp=768, magnitude_type="cosine"),
    "small_random_sep": dict(layer="ConvNNAttention", num_heads=1, d_hidden=384, d_mlp=1536, magnitude_type="euclidean",
                             sampling_type="random", num_samples=40, convolution_type="depthwise-separable"),
    "spatial_coord": dict(layer="ConvNNAttention", num_heads=3, d_hidden=96, d_mlp=200, sampling_type="spatial",
                          num_samples=50, convolution_type="standard", coordinate_encoding=True),
    "branch_attention": dict(layer="BranchAttention", num_heads=3, d_hidden=192, d_mlp=768),
    "branch_conv": dict(layer="BranchConv", num_heads=3, d_hidden=192, d_mlp=768, kernel_size=5),
}


def _model(cfg, dtype, seed=0):
    torch.manual_seed(seed)
    m = convnn_b200.ViT(convnn_b200.make_args(num_layers=3, dropout=0.0, attention_dropout=0.0, num_classes=24, device=DEV,
                                              **CONFIGS[cfg])).to(dtype).eval()
    if m.args.sampling_type == "random":
        m.set_candidates(torch.randperm(197)[:40])
    return m


def _op_by_op(model, x):
    model_plan._plans.pop(model, None)
    y = model(x)                                  # the first call of a shape takes the op-by-op path
    return y


def _planned(model, x):
    for _ in range(2):
        model(x)
    plan = model_plan._plans[model][(x.shape, x.dtype, x.device)]
    assert type(plan) is model_plan.Plan
    return model(x)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("cfg", sorted(CONFIGS))
def test_plan_gives_the_same_bits(cfg, dtype):
    m = _model(cfg, dtype)
    with torch.no_grad():
        for B in (1, 5):
            x = torch.randn(B, 3, 224, 224, device=DEV).to(dtype)
            assert torch.equal(_op_by_op(m, x), _planned(m, x))
        u8 = torch.randint(0, 256, (2, 3, 224, 224), device=DEV, dtype=torch.uint8)
        assert torch.equal(_op_by_op(m, u8), _planned(m, u8))


def test_plan_follows_changes_of_the_model():
    m = _model("tiny", torch.bfloat16)
    x = torch.randn(2, 3, 224, 224, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        before = _planned(m, x)
        changes = [
            lambda: m.transformer_encoder[1].mlp[0].weight.mul_(1.5),                          # in place
            lambda: setattr(m.classifier, "weight", torch.nn.Parameter(m.classifier.weight * 2)),  # replaced
            lambda: setattr(m.transformer_encoder[0].attention, "magnitude_type", "matmul"),   # option of a layer
            lambda: m.transformer_encoder.__setitem__(2, copy.deepcopy(m.transformer_encoder[0])),  # module of the tree
            lambda: setattr(m.transformer_encoder[0], "fold_layernorm", False),
        ]
        for change in changes:
            change()
            got = m(x)
            want = _op_by_op(m, x)
            assert torch.equal(got, want) and not torch.equal(got, before)
            before = _planned(m, x)
            assert torch.equal(before, want)
        seen = []                                 # (hooks of the modules that are called take the op-by-op path)
        m.transformer_encoder[0].fold_layernorm = False
        m.transformer_encoder[0].attention.register_forward_hook(lambda *a: seen.append(len(a)))
        outs = [m(x) for _ in range(4)]
        assert len(seen) == 4 and all(torch.equal(y, _op_by_op(m, x)) for y in outs)


def test_random_candidates_are_drawn_per_call_as_before():
    m = _model("small_random_sep", torch.float32)
    m.set_candidates(None)
    x = torch.randn(2, 3, 224, 224, device=DEV)
    with torch.no_grad():
        torch.manual_seed(5)
        want = [_op_by_op(m, x), _op_by_op(m, x)]
        _planned(m, x)
        torch.manual_seed(5)
        assert all(torch.equal(m(x), w) for w in want)


def test_layer_call_follows_changes_and_options():
    torch.manual_seed(1)
    m = convnn_b200.MultiHeadConvNNAttention(96, 3, 0.0, 9, "spatial", 50, 0, "cosine").to(DEV, torch.bfloat16).eval()
    x = torch.randn(2, 197, 96, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        first = m(x)
        assert torch.equal(m(x), first) and len(m._calls) == 1
        wide = torch.zeros(2, 197, 200, device=DEV, dtype=torch.bfloat16)
        assert torch.equal(m(x, out=wide[:, :, 8:104], residual=x), first + x) and torch.equal(wide[:, :, 8:104], first + x)
        m.W_v.weight.mul_(2.0)
        assert not torch.equal(m(x), first)
        fresh = copy.deepcopy(m)
        assert len(fresh._calls) == 0 and torch.equal(fresh(x), m(x))
        m.K = 5                                   # an option of the layer, with taps cut to it
        m.conv.weight.data = m.conv.weight.data[:, :, :5].contiguous()
        short = convnn_b200.MultiHeadConvNNAttention(96, 3, 0.0, 5, "spatial", 50, 0, "cosine").to(DEV, torch.bfloat16).eval()
        short.load_state_dict(m.state_dict())
        assert torch.equal(m(x), short(x)) and not torch.equal(m(x), fresh(x))
        m.magnitude_type = "unknown"
        with pytest.raises(ValueError, match="magnitude_type"):
            m(x)


@pytest.mark.parametrize("cfg", sorted(CONFIGS))
def test_weights_written_by_the_launch_before_a_forward(cfg):
    """Weights changed in stream order, without a wait, by other kernels than the library's: turn by turn the op-by-op path and a
    new plan.  (Weights written by a library kernel that lets the next one start early: test_gpu_launch_order.py.)"""
    m = _model(cfg, torch.bfloat16)
    x = torch.randn(3, 3, 224, 224, device=DEV).bfloat16()
    kept = [{n: p.detach() * f for n, p in m.named_parameters()} for f in (0.5, 1.5, 1.0)]
    with torch.no_grad():
        want = []
        for w in kept:
            for n, p in m.named_parameters():
                p.copy_(w[n])
            torch.cuda.synchronize()
            want.append(_op_by_op(m, x))
        for _ in range(2):
            m(x)
        for turn in range(12):
            for n, p in m.named_parameters():
                p.copy_(kept[turn % 3][n])
            assert torch.equal(m(x), want[turn % 3])


@pytest.mark.parametrize("heads,conv", [(3, "depthwise"), (3, "standard"), (1, "depthwise"), (1, "depthwise-separable")])
@pytest.mark.parametrize("layer", ["BranchConv", "BranchAttention"])
@pytest.mark.parametrize("B", [1, 5, 40])
def test_halves_side_by_side_give_the_bits_of_one_after_the_other(layer, heads, conv, B):
    """A branching block's halves run beside each other where the workspace has room for both; one page less, and they do not."""
    torch.manual_seed(3)
    m = convnn_b200.ViT(convnn_b200.make_args(layer=layer, num_layers=4, num_heads=heads, d_hidden=192, d_mlp=768, dropout=0.0,
                                              attention_dropout=0.0, num_classes=24, convolution_type=conv,
                                              device=DEV)).to(torch.bfloat16).eval()
    x = torch.randn(B, 3, 224, 224, device=DEV).bfloat16()
    with torch.no_grad():
        want = _op_by_op(m, x)
        got = [_planned(m, x) for _ in range(20)]
        plan = model_plan._plans[m][(x.shape, x.dtype, x.device)]
        plan.workspace_bytes -= 256
        got += [m(x) for _ in range(3)]
        assert model_plan._plans[m][(x.shape, x.dtype, x.device)] is plan
    assert all(torch.equal(y, want) for y in got)


@pytest.mark.parametrize("layer", ["BranchConv", "BranchAttention"])
def test_no_room_for_both_halves(layer, monkeypatch):
    """Memory for one half of a branching block at a time is enough, as before the halves ran side by side."""
    torch.manual_seed(3)
    m = convnn_b200.ViT(convnn_b200.make_args(layer=layer, num_layers=3, num_heads=3, d_hidden=192, d_mlp=768, dropout=0.0,
                                              attention_dropout=0.0, num_classes=24, device=DEV)).to(torch.bfloat16).eval()
    x = torch.randn(5, 3, 224, 224, device=DEV).bfloat16()
    allocate = torch.empty

    def limited(*size, **kw):
        if kw.get("dtype") is torch.uint8 and size[0] > plan.least_bytes:
            raise torch.cuda.OutOfMemoryError("out of memory")
        return allocate(*size, **kw)

    with torch.no_grad():
        want = _planned(m, x)
        plan = model_plan._plans[m][(x.shape, x.dtype, x.device)]
        assert 0 < plan.least_bytes < plan.workspace_bytes
        monkeypatch.setattr(torch, "empty", limited)
        got = [m(x) for _ in range(3)]
        monkeypatch.undo()
        assert model_plan._plans[m][(x.shape, x.dtype, x.device)] is plan
    assert all(torch.equal(y, want) for y in got)
