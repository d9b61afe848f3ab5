"""CUDA graphs and streams around what the host side keeps between forwards: a graph must not read anything that is gone
or was written elsewhere by the time it is replayed."""
import pytest
import torch

import convnn_b200
from convnn_b200 import model_plan

pytestmark = pytest.mark.gpu
DEV = "cuda"
SETS = ["override", "host", "spatial"]


def _model(kind):
    torch.manual_seed(0)
    m = convnn_b200.ViT(convnn_b200.make_args(
        num_layers=2, num_heads=1, d_hidden=64, d_mlp=128, num_classes=24, device=DEV, dropout=0.0, attention_dropout=0.0,
        magnitude_type="cosine", sampling_type="spatial" if kind == "spatial" else "random", num_samples=40))
    m = m.to(torch.bfloat16).eval()
    if kind != "spatial":
        m.set_candidates(torch.randperm(197, device=DEV if kind == "override" else "cpu")[:40])
    return m


def _layer(kind):
    torch.manual_seed(0)
    m = convnn_b200.MultiHeadConvNNAttention(64, 1, 0.0, 9, "spatial" if kind == "spatial" else "random", 40, 0, "cosine")
    m = m.to(DEV, torch.bfloat16).eval()
    if kind != "spatial":
        m.candidate_override = torch.randperm(197, device=DEV if kind == "override" else "cpu")[:40]
    return m


def _case(which, kind):
    return (_model(kind), (3, 3, 224, 224)) if which == "vit" else (_layer(kind), (3, 197, 64))


def _drop(m):
    """What building another model, a change of this one, or more shapes than are remembered does to a shape's entry."""
    model_plan._plans.pop(m, None)
    getattr(m, "_calls", {}).clear()


@pytest.mark.parametrize("kind", SETS)
@pytest.mark.parametrize("which", ["vit", "layer"])
@torch.no_grad()
def test_graph_outlives_what_it_was_captured_with(which, kind):
    m, shape = _case(which, kind)
    x = torch.randn(shape, device=DEV).bfloat16()
    for _ in range(3):
        want = m(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = m(x)
    _drop(m)
    keep = [torch.zeros(n, dtype=torch.int32, device=DEV) for n in [40, 64, 128, 256] * 200]    # takes over freed memory
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and len(keep) == 800


@pytest.mark.parametrize("which", ["vit", "layer"])
@torch.no_grad()
def test_graph_follows_candidates_changed_between_replays(which):
    m, shape = _case(which, "override")
    x = torch.randn(shape, device=DEV).bfloat16()
    for _ in range(3):
        m(x)
    first = m.candidate_override if which == "layer" else m.transformer_encoder[0].attention.candidate_override
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = m(x)
    first.copy_(torch.randperm(197, device=DEV)[:40])
    g.replay()
    got = y.clone()
    assert torch.equal(got, m(x))


@pytest.mark.parametrize("kind", SETS)
@pytest.mark.parametrize("which", ["vit", "layer"])
@torch.no_grad()
def test_another_stream_reads_nothing_unfinished(which, kind):
    m, shape = _case(which, kind)
    x = torch.randn(shape, device=DEV).bfloat16()
    want = m(x)
    torch.cuda.synchronize()
    other = torch.cuda.Stream()
    torch.cuda._sleep(20_000_000)                 # the current stream is busy: its work so far is not done
    m(x)                                          # prepares what a shape keeps
    with torch.cuda.stream(other):
        y = m(x)
    other.synchronize()
    assert torch.equal(y, want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("kind", SETS)
@pytest.mark.parametrize("which", ["vit", "layer"])
@torch.no_grad()
def test_one_warm_up_then_capture_then_an_eager_call(which, kind):
    m, shape = _case(which, kind)
    x = torch.randn(shape, device=DEV).bfloat16()
    want = m(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = m(x)
    for _ in range(3):                            # before any replay: nothing recorded has run
        assert torch.equal(m(x), want)
    g.replay()
    assert torch.equal(y, want)


@pytest.mark.parametrize("which", ["vit", "layer"])
@torch.no_grad()
def test_deleted_model_gives_its_memory_back(which):
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    m, shape = _case(which, "spatial")
    x = torch.randn(shape, device=DEV).bfloat16()
    for _ in range(3):
        m(x)
    torch.cuda.synchronize()
    del m, x
    assert torch.cuda.memory_allocated() == before


@pytest.mark.parametrize("which", ["vit", "layer"])
@torch.no_grad()
def test_host_set_changed_in_place(which):
    """Followed by later calls; a graph keeps what it was captured with, also when its copy has been replaced."""
    m, shape = _case(which, "host")
    x = torch.randn(shape, device=DEV).bfloat16()
    cand = m.candidate_override if which == "layer" else m.transformer_encoder[0].attention.candidate_override
    for _ in range(3):
        first = m(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = m(x)
    for seed in (1, 2):
        cand.copy_(torch.randperm(197, generator=torch.Generator().manual_seed(seed))[:40])
        got = [m(x) for _ in range(3)]
        _drop(m)
        assert all(torch.equal(a, m(x)) for a in got) and not torch.equal(got[0], first)
    keep = [torch.zeros(n, dtype=torch.int32, device=DEV) for n in [40, 64, 128, 256] * 200]
    g.replay()
    assert torch.equal(y, first) and len(keep) == 800
