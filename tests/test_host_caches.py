"""What the host side keeps between forwards (the ViT's host plan, the layers' prepared calls), on CPU tensors: the
native entry points are replaced by recorders of what they are handed."""
import copy
import ctypes
import gc
import pickle
import threading
import types
import weakref

import numpy as np
import pytest
import torch

import convnn_b200
from convnn_b200 import _capi, layers, model_plan, ops


def _ints(pointer, n):
    return list((ctypes.c_int32 * n).from_address(pointer)) if pointer else None


@pytest.fixture
def host(monkeypatch):
    """The host path on CPU; ``host.models`` / ``host.layers`` list the recorded native calls."""
    rec = types.SimpleNamespace(models=[], layers=[], general=[])
    lib = _capi.lib()

    def model_forward(arg, images, logits, workspace, nbytes, stream):
        m = arg._obj
        rec.models.append(types.SimpleNamespace(
            embed_eps=m.embed_eps, eps=[(b.eps1, b.eps2) for b in m.blocks[:m.n_blocks]],
            cand=[_ints(b.cand, b.layer.S) if b.layer.sampled else None for b in m.blocks[:m.n_blocks]],
            cand_ptr=[b.cand for b in m.blocks[:m.n_blocks]], pixel_mean=m.pixel_mean))
        return 0

    def layer_forward(d, x, ldx, w_qkv, w_conv, w_pw, w_o, cand, *rest):
        rec.layers.append(types.SimpleNamespace(cand=_ints(cand, d.S) if d.sampled else None, w_pw=w_pw, w_conv=w_conv,
                                                ldo=rest[3], K=d.K))
        return 0
    monkeypatch.setattr(lib, "convnn_b200_model_forward", model_forward)
    monkeypatch.setattr(lib, "convnn_b200_forward", layer_forward)
    monkeypatch.setattr(ops, "_stream", lambda t: 0)
    monkeypatch.setattr(ops, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(layers.MultiHeadConvNNAttention, "_check_mode", lambda self, x: None)
    return rec


def _vit(**kw):
    args = dict(img_size=(3, 32, 32), patch_size=8, num_layers=2, num_heads=1, d_hidden=16, d_mlp=32, num_classes=5, K=3,
                magnitude_type="cosine", dropout=0.0, attention_dropout=0.0, device="cpu")
    args.update(kw)
    return convnn_b200.ViT(convnn_b200.make_args(**args)).eval()


def _layer(*, K=3, conv="depthwise", sampling="all", samples=-1):
    return convnn_b200.MultiHeadConvNNAttention(16, 1, 0.0, K, sampling, samples, 0, "cosine", convolution_type=conv).eval()


def _images(B=2):
    return torch.randn(B, 3, 32, 32)


@torch.no_grad()
def test_plan_takes_the_candidates_of_each_call(host):
    m, x = _vit(sampling_type="random", num_samples=6), _images()
    numbers = np.arange(6)
    m.set_candidates(torch.from_numpy(numbers))
    for _ in range(3):
        model_plan.run(m, x)
    assert host.models[-1].cand == [list(range(6))] * 2
    numbers += 7                                  # in place, where no version counter sees it
    model_plan.run(m, x)
    assert host.models[-1].cand == [list(range(7, 13))] * 2


@torch.no_grad()
def test_layer_call_takes_the_candidates_of_each_call(host):
    m, x = _layer(sampling="random", samples=6), torch.randn(2, 17, 16)
    numbers = np.arange(6)
    m.candidate_override = torch.from_numpy(numbers)
    for _ in range(3):
        m(x)
    numbers += 7
    m(x)
    assert host.layers[-1].cand == list(range(7, 13))


@torch.no_grad()
def test_candidates_of_another_size(host):
    m, x = _vit(sampling_type="random", num_samples=6), _images()
    cand = torch.arange(6)
    m.set_candidates(cand)
    for _ in range(2):
        model_plan.run(m, x)
    cand.set_(torch.arange(9))
    for _ in range(3):                            # op by op, noticed, planned again
        model_plan.run(m, x)
    assert host.models[-1].cand == [list(range(9))] * 2
    lay = _layer(sampling="random", samples=6)
    lay.candidate_override = cand = torch.arange(6)
    lx = torch.randn(2, 17, 16)
    for _ in range(2):
        lay(lx)
    cand.set_(torch.arange(9))
    lay(lx)
    assert host.layers[-1].cand == list(range(9))


@torch.no_grad()
def test_spatial_candidates_belong_to_the_layer(host):
    m, x = _vit(sampling_type="spatial", num_samples=5), _images()
    for _ in range(2):
        model_plan.run(m, x)
    want = torch.linspace(0, 16, 5).long().tolist()
    assert host.models[-1].cand == [want] * 2
    before = host.models[-1].cand_ptr
    model_plan._plans.pop(m)                       # a captured graph outlives the plan it was captured with
    for _ in range(2):
        model_plan.run(m, x)
    assert host.models[-1].cand_ptr == before


@torch.no_grad()
def test_nothing_is_prepared_while_a_graph_is_captured(host, monkeypatch):
    m, x = _vit(sampling_type="spatial", num_samples=5), _images()
    lay, lx = _layer(sampling="spatial", samples=5), torch.randn(2, 17, 16)
    model_plan.run(m, x), lay(lx)
    monkeypatch.setattr(layers, "capturing", lambda device: True)
    assert model_plan.run(m, x) is None and not host.models
    lay(lx)
    assert len(host.layers) == 2 and not lay._calls
    monkeypatch.setattr(layers, "capturing", lambda device: False)
    model_plan.run(m, x), lay(lx)
    assert len(host.models) == 1 and len(lay._calls) == 1
    monkeypatch.setattr(layers, "capturing", lambda device: True)
    model_plan.run(m, x), lay(lx)                  # what is there already serves a capture too
    assert len(host.models) == 2 and len(host.layers) == 4


def test_spatial_set_of_a_capture_is_not_kept(monkeypatch):
    lay = _layer(sampling="spatial", samples=5)
    monkeypatch.setattr(layers, "capturing", lambda device: True)
    assert lay.candidates(17, torch.device("cpu")).tolist() == [0, 4, 8, 12, 16] and not lay._spatial_cache
    assert lay.kernel_candidates(17, torch.device("cpu")).tolist() == [0, 4, 8, 12, 16] and not lay._spatial_cache
    monkeypatch.setattr(layers, "capturing", lambda device: False)
    assert lay.kernel_candidates(17, torch.device("cpu")).tolist() == [0, 4, 8, 12, 16] and len(lay._spatial_cache) == 2


@torch.no_grad()
def test_models_and_layers_are_freed(host):
    """By their last reference, not by a later collection: their weights are GPU memory."""
    m, x = _vit(sampling_type="random", num_samples=6), _images()
    for _ in range(3):
        model_plan.run(m, x)
    lay, lx = _layer(sampling="random", samples=6), torch.randn(2, 17, 16)
    for _ in range(3):
        lay(lx)
    assert len(host.models) == 2 and len(lay._calls) == 1
    dead = [weakref.ref(o) for o in (m, m.classifier.weight, lay, lay.W_v.weight)]
    plans = len(model_plan._plans)
    gc.disable()
    try:
        del m, lay
        assert [r() for r in dead] == [None] * 4 and len(model_plan._plans) == plans - 1
    finally:
        gc.enable()


@torch.no_grad()
def test_packed_weights_of_another_parameter_version_are_given_back(host):
    lay, m = _layer(), _vit()
    for B in (1, 2, 3):
        for _ in range(2):
            lay(torch.randn(B, 17, 16)), model_plan.run(m, _images(B))
    att = m.transformer_encoder[0].attention
    old = [weakref.ref(w) for w in lay._packed + att._packed if w is not None]
    for layer in (lay, att):
        layer.W_v.weight.mul_(2.0)
    for _ in range(2):
        lay(torch.randn(2, 17, 16)), model_plan.run(m, _images(2))
    gc.collect()
    assert all(r() is None for r in old)


@torch.no_grad()
def test_plan_follows_the_eps_of_the_norms(host):
    m, x = _vit(), _images()
    for _ in range(2):
        model_plan.run(m, x)
    m.transformer_encoder[0].norm1.eps = 0.5
    m.transformer_encoder[1].norm2.eps = 0.25
    m.patch_embedding.norm.eps = 0.125
    for _ in range(2):
        model_plan.run(m, x)
    last = host.models[-1]
    assert last.eps[0][0] == 0.5 and last.eps[1][1] == 0.25 and last.embed_eps == 0.125


@torch.no_grad()
def test_plan_follows_the_patch_size_it_was_given(host):
    m, x = _vit(), _images()
    for _ in range(2):
        model_plan.run(m, x)
    m.args.patch_size = 4                          # no longer what the weights are for: the op-by-op path refuses it
    assert model_plan.run(m, x) is None


@torch.no_grad()
def test_layer_call_follows_its_modules(host):
    lay, x = _layer(conv="depthwise-separable"), torch.randn(2, 17, 16)
    for _ in range(3):
        lay(x)
    old = host.layers[-1]
    lay.conv[1] = torch.nn.Conv1d(16, 16, 1, bias=False)
    lay(x)
    torch.testing.assert_close(lay._packed[2], lay.conv[1].weight[:, :, 0])
    new = host.layers[-1]
    assert new.w_pw == lay._packed[2].data_ptr() and new.w_pw != old.w_pw


@torch.no_grad()
def test_plan_follows_the_pixel_statistics(host):
    m, x = _vit(), torch.randint(0, 256, (2, 3, 32, 32), dtype=torch.uint8)
    m.pixel_mean = [0.5, 0.5, 0.5]
    for _ in range(3):
        model_plan.run(m, x)
    assert host.models[-1].pixel_mean == m.pixel_stats(x.device)[1].data_ptr()
    m.pixel_mean[1] = 0.25                         # in place: no assignment to count
    for _ in range(2):
        model_plan.run(m, x)
    now = m.pixel_stats(x.device)[1]
    assert now.tolist() == [0.5, 0.25, 0.5] and host.models[-1].pixel_mean == now.data_ptr()


def test_tensors_made_under_inference_mode(host):
    """They have no version counter: a converted model's buffers, a candidate set."""
    m, x = _vit(sampling_type="random", num_samples=6), _images()
    with torch.inference_mode():
        m = m.double().float()
        m.set_candidates(torch.randperm(17)[:6])
    lay, lx = _layer(sampling="random", samples=6), torch.randn(2, 17, 16)
    with torch.inference_mode():
        lay.candidate_override = torch.arange(6)
    with pytest.raises(RuntimeError):
        m.positional_encoding.pe._version
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            for _ in range(3):
                model_plan.run(m, x), lay(lx)
    assert len(host.models) == 5 and len(host.layers) == 6


@torch.no_grad()
def test_plans_outlive_assignments_that_do_not_concern_them(host):
    m, x = _vit(), _images()
    lay, lx = _layer(), torch.randn(2, 17, 16)
    for _ in range(2):
        model_plan.run(m, x), lay(lx)
    plan, call = next(iter(model_plan._plans[m].values())), next(iter(lay._calls.values()))
    _vit().classifier.bias.zero_()                 # another model is built
    _layer().K = 2                                 # and changed
    for _ in range(3):
        m.eval(), lay.eval()                       # nothing changes
        assert model_plan.run(m, x) is not None and lay(lx) is not None
    assert next(iter(model_plan._plans[m].values())) is plan and next(iter(lay._calls.values())) is call
    lay.train()
    lay.softmax_topk_val = False
    lay.eval(), lay(lx)
    assert next(iter(lay._calls.values())) is not call
    m.transformer_encoder[1].attention.softmax_topk_val = False
    assert model_plan.run(m, x) is None


@torch.no_grad()
def test_twenty_batch_sizes_keep_their_plans(host):
    m = _vit()
    for turn in range(4):
        for B in range(1, 21):
            assert (model_plan.run(m, _images(B)) is not None) == (turn > 0)
    assert len(model_plan._plans[m]) == 20
    for B in range(21, 21 + model_plan.MAX_PLANS):  # bounded, and those in use stay
        model_plan.run(m, _images(1)), model_plan.run(m, _images(B))
    assert len(model_plan._plans[m]) == model_plan.MAX_PLANS and model_plan.run(m, _images(1)) is not None


@torch.no_grad()
def test_plans_of_a_model_from_many_threads(host, monkeypatch):
    m, failures = _vit(), []
    monkeypatch.setattr(model_plan, "MAX_PLANS", 3)

    def work(seed):
        try:
            for i in range(60):
                model_plan.run(m, _images(1 + (i * seed) % 7))
        except Exception as e:                     # noqa: BLE001
            failures.append(e)
    with torch.no_grad():
        threads = [threading.Thread(target=torch.no_grad()(work), args=(s,)) for s in (1, 2, 3, 5)]
        [t.start() for t in threads], [t.join() for t in threads]
    assert not failures and len(model_plan._plans[m]) <= 3


@torch.no_grad()
def test_calls_that_run_somebody_elses_code_are_not_planned(host):
    """The op-by-op path calls a block's attention, and the halves of a branching one, as modules; they may be a subclass or
    have a forward of their own.  Weights that are no registered parameters cannot be watched."""
    class Mine(layers.MultiHeadAttention):
        pass

    def own_forward(m):
        m.transformer_encoder[1].attention.forward = lambda x, residual=None: residual

    def own_half(m):
        att = m.transformer_encoder[0].attention
        att.attention = Mine(att.d_hidden_attention, att.num_heads, 0.0).eval()

    def own_forward_of_a_half(m):
        m.transformer_encoder[0].attention.convnn.forward = lambda x, out=None: out

    def plain_weight(m):
        lin = m.transformer_encoder[1].mlp[0]
        w = lin.weight.detach().clone()
        del lin.weight
        lin.weight = w

    def plain_packed_weight(m):
        lin = m.transformer_encoder[1].attention.convnn.W_v
        w = lin.weight.detach().clone()
        del lin.weight
        lin.weight = w

    x = _images()
    for change in (own_forward, own_half, own_forward_of_a_half, plain_weight, plain_packed_weight):
        m = _vit(layer="BranchAttention", d_hidden=32)
        for _ in range(2):
            model_plan.run(m, x)
        assert host.models
        host.models.clear()
        change(m)
        assert [model_plan.run(m, x) for _ in range(4)] == [None] * 4 and not host.models, change.__name__
    lay, lx = _layer(), torch.randn(2, 17, 16)
    w = lay.W_v.weight.detach().clone()
    del lay.W_v.weight
    lay.W_v.weight = w
    lay(lx), lay(lx)
    lay.W_v.weight = w * 2
    lay(lx)
    torch.testing.assert_close(lay._packed[0][1], w * 2)


@torch.no_grad()
def test_input_of_another_width_than_the_layer(host):
    """The result has rows as wide as the input's, and the library is told so (it refuses rows narrower than the layer:
    a channel slice that is too narrow must not be written past its rows)."""
    for x in (torch.randn(2, 17, 24), torch.randn(2, 17, 24)[:, :, :8]):
        lay = _layer()
        seen = [(lay(x).shape, host.layers[-1].ldo) for _ in range(3)]
        assert seen == [(x.shape, x.shape[2])] * 3


@torch.no_grad()
def test_modules_saved_before_they_kept_prepared_calls(host):
    lay, x = _layer(), torch.randn(2, 17, 16)
    old = copy.deepcopy(lay)
    old(x)
    for name in ("_calls", "_stamp"):
        old.__dict__.pop(name)
    old = pickle.loads(pickle.dumps(old))
    for _ in range(3):
        old(x)
    assert len(host.layers) == 4
    new = pickle.loads(pickle.dumps(lay))
    new(x), new(x)
    assert len(new._calls) == 1
