"""Helpers shared by the GPU parity tests: every CUDA result is obtained through the C ABI
(convnn_b200.ops / the nn.Modules) and compared with the CPU oracle."""
import pytest
import torch

import convnn_b200
from convnn_b200 import ops
from oracle.convnn_oracle import ConvNNConfig

DEV = "cuda"

# tests of a dispatch that goes by the number of SMs
on_148_sms = pytest.mark.skipif(torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != 148,
                                reason="the lines of this rule are tested for 148 SMs")


def spec_of(cfg: ConvNNConfig) -> ops.LayerSpec:
    return ops.LayerSpec(cfg.d_hidden, cfg.num_heads, cfg.K, cfg.sampling_type, cfg.magnitude_type,
                         cfg.convolution_type, cfg.softmax_topk_val, cfg.coordinate_encoding, cfg.seq_length)


def conv_params(cfg, w):
    if cfg.convolution_type == "depthwise-separable":
        return (w["conv.0.weight"], w["conv.1.weight"])
    return (w["conv.weight"],)


def pack(cfg, w, dtype):
    return ops.pack_weights(spec_of(cfg), w["W_q.weight"], w["W_k.weight"], w["W_v.weight"], w["W_o.weight"],
                            conv_params(cfg, w), dtype, torch.device(DEV))


def module_of(cfg: ConvNNConfig, w, dtype):
    m = convnn_b200.MultiHeadConvNNAttention(
        cfg.d_hidden, cfg.num_heads, 0.0, cfg.K, cfg.sampling_type, cfg.num_samples, cfg.sample_padding,
        cfg.magnitude_type, cfg.seq_length, cfg.coordinate_encoding, cfg.convolution_type, cfg.softmax_topk_val)
    m.load_state_dict(w, strict=True)
    return m.eval().to(DEV, dtype)


def heads_to_oracle(t, C):
    """(B, R, H, Cp) device tensor -> (B, H, R, C) float32 CPU (oracle layout)."""
    return t[..., :C].permute(0, 2, 1, 3).float().cpu().contiguous()


def rel_err(a, b):
    a, b = a.double().cpu(), b.double().cpu()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def launches(fn, attribute="LOCAL_SIZE_BYTES"):
    """{kernel name (mangled): bytes of local memory per thread, or another attribute, or its CTAs ("GRID")} of what fn() launches,
    read from a captured graph."""
    from cuda.bindings import driver

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1:]

    fn()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        fn()
    raw = driver.CUgraph(graph.raw_cuda_graph())
    count = ok(driver.cuGraphGetNodes(raw, 0))[-1]
    found = {}
    for node in ok(driver.cuGraphGetNodes(raw, count))[0][:count]:
        if ok(driver.cuGraphNodeGetType(node))[0] != driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        p = ok(driver.cuGraphKernelNodeGetParams(node))[0]
        func = p.func if int(p.func) else ok(driver.cuKernelGetFunction(p.kern))[0]
        name = ok(driver.cuFuncGetName(func))[0].decode()
        found[name] = p.gridDimX * p.gridDimY * p.gridDimZ if attribute == "GRID" else ok(driver.cuFuncGetAttribute(
            getattr(driver.CUfunction_attribute, "CU_FUNC_ATTRIBUTE_" + attribute), func))[0]
    graph.reset()
    return found
