"""Drop-in ``nn.Module``s for the reference's ConvNN-Attention layers.

Same constructor arguments, ``state_dict`` keys and ``forward(x)`` signature as
``MultiHeadConvNNAttention`` (reference layers.py:132-321), ``MultiHeadBranchingAttention``
(layers.py:580-652) and ``MultiHeadBranchingConv`` (layers.py:502-578), so a reference
checkpoint loads with ``strict=True`` and the reference's ``vit.py`` can construct them
in place of its own.  The ConvNN path runs in libconvnn_b200 (CUDA, sm_100a); it is
forward-only (inference) and has no CPU implementation.  The other halves of the branching
wrappers (softmax attention, Conv1d attention) and ``pointwise_linear`` run in the same
library; their modules only hold the parameters under the reference's names.
"""
from __future__ import annotations

import itertools
from typing import Optional

import torch
import torch.nn as nn

from . import ops
from .ops import LayerSpec


_stamps = itertools.count(1)
_ABSENT = object()
_PLAIN = (bool, int, float, str, tuple, type(None))


class WatchedModule(nn.Module):
    """``nn.Module`` that gets a new ``_stamp`` whenever a public attribute is given another value: whatever was prepared
    from its attributes (a forward's host plan) is valid while the stamp stands.  The stamp comes after the assignment, so
    what another thread prepares in between is at worst prepared again."""

    def __setattr__(self, name, value):
        old = self.__dict__.get(name, _ABSENT)
        super().__setattr__(name, value)
        if name[0] != "_" and not (old is value and type(value) in _PLAIN):
            self.__dict__["_stamp"] = next(_stamps)

    def __delattr__(self, name):
        super().__delattr__(name)
        self.__dict__["_stamp"] = next(_stamps)


def capturing(device) -> bool:
    """Whether work on a CUDA ``device`` is being recorded into a graph.  What such work writes does not exist before the
    first replay, so nothing prepared in it is kept for later calls."""
    return device.type == "cuda" and torch.cuda.is_current_stream_capturing()


class _NotCopied(dict):
    """A cache that copies and pickles of its owner start without."""

    def __deepcopy__(self, memo):
        return _NotCopied()

    def __reduce__(self):
        return (_NotCopied, ())


def _counts_versions(t) -> bool:
    """False for tensors made under ``torch.inference_mode()``."""
    try:
        return t._version >= 0
    except RuntimeError:
        return False


class Watch:
    """The state of ``root`` and the modules below it that something prepared is valid for: one walk, taken before the
    preparation.  It holds the modules below ``root`` but not ``root``, which owns what was prepared and must not be kept
    alive by it."""

    def __init__(self, root):
        self.mods, self.trees, self.slots, self.tensors, self.hooks = [], [], [], [], []
        todo, seen = [root], set()
        while todo:
            m = todo.pop()
            if m is None or id(m) in seen:
                continue
            seen.add(id(m))
            d = m.__dict__
            if m is not root:
                self.mods.append(m)
            children = d["_modules"]
            if children:
                self.trees.append((children, dict(children)))
                todo.extend(children.values())
            self.hooks += (d["_forward_hooks"], d["_forward_pre_hooks"])
            for tensors in (d["_parameters"], d["_buffers"]):
                for k, t in tensors.items():
                    self.slots.append((tensors, k))
                    if t is not None:
                        self.tensors.append(t)
        self.dicts = [m.__dict__ for m in self.mods if isinstance(m, WatchedModule)]
        self.stamps = self._stamps(root)
        self.ids = [id(d[k]) for d, k in self.slots]
        # (what is packed from a tensor without a version counter is refused where it is packed; others are read in place)
        self.versioned = [t for t in self.tensors if _counts_versions(t)]
        self.versions = [t._version for t in self.versioned]
        self.ptrs = [t.data_ptr() for t in self.tensors]

    def _stamps(self, root):
        return [d.get("_stamp") for d in self.dicts] + [root.__dict__.get("_stamp")]

    def options_unchanged(self, root) -> bool:
        return self._stamps(root) == self.stamps

    def unchanged(self, root) -> bool:
        return (self._stamps(root) == self.stamps and
                [id(d[k]) for d, k in self.slots if k in d] == self.ids and
                [t._version for t in self.versioned] == self.versions and
                [t.data_ptr() for t in self.tensors] == self.ptrs and
                all([d == c for d, c in self.trees]))


def registered(*modules) -> bool:
    """Whether the weights and biases of ``modules`` are parameters, which a ``Watch`` sees (and no attributes or
    parametrizations)."""
    return all(m._parameters.keys() >= {"weight", "bias"} for m in modules)


class _LayerCall:
    """What one ConvNN layer call of a given input shape needs besides its tensors, prepared once: descriptor, packed
    weights, workspace size (27 us of host time per call before, 10 with it; a small layer's kernels take 30).
    Candidates are not part of it (``kernel_candidates``): a captured graph would read them after this object is gone."""

    def __init__(self, layer, x):
        B, T, _ = x.shape
        self.watch = Watch(layer)
        self.S = layer.candidate_count(T, x.device)
        self.packed = layer.packed_weights(x.dtype, x.device)
        self.call = ops.LayerForward(layer._spec(), B, T, self.S, x.dtype, x.device, self.packed)

    def __call__(self, layer, x, out, residual):
        """``layer(x)``; None: the candidate set has another size now."""
        cand = layer.kernel_candidates(x.shape[1], x.device)
        if cand is not None and cand.numel() != self.S:
            return None
        return self.call(x, cand, out, residual)


class MultiHeadConvNNAttention(WatchedModule):
    def __init__(self, d_hidden, num_heads, attention_dropout, K, sampling_type, num_samples, sample_padding,
                 magnitude_type, seq_length=197, coordinate_encoding=False, convolution_type='depthwise',
                 softmax_topk_val=True):
        super().__init__()
        assert d_hidden % num_heads == 0, "d_hidden must be divisible by num_heads"
        self.d_hidden = d_hidden
        self.num_heads = num_heads
        self.attention_dropout = attention_dropout
        self.d_k = d_hidden // num_heads
        self.K = K
        self.seq_length = seq_length
        self.sampling_type = sampling_type
        self.num_samples = int(num_samples)
        self.sample_padding = int(sample_padding) if sampling_type == 'spatial' else 0
        self.magnitude_type = magnitude_type
        self.maximum = magnitude_type in ('cosine', 'matmul')
        self.coordinate_encoding = coordinate_encoding
        self.convolution_type = convolution_type
        self.softmax_topk_val = softmax_topk_val
        self.INF = 1.1
        self.NEG_INF = -0.1

        self.W_q = nn.Linear(d_hidden, d_hidden, bias=False)
        self.W_k = nn.Linear(d_hidden, d_hidden, bias=False)
        self.W_v = nn.Linear(d_hidden, d_hidden, bias=False)
        self.W_o = nn.Linear(d_hidden, d_hidden, bias=False)
        self.dropout = nn.Dropout(attention_dropout)

        self.in_channels = self.d_k + 1 if coordinate_encoding else self.d_k
        self.out_channels = self.d_k
        C, dk = self.in_channels, self.d_k
        # Parameter containers only (never called): they give the reference's state_dict
        # keys and its construction-time errors, e.g. depthwise + coordinate_encoding.
        if convolution_type == 'standard':
            self.conv = nn.Conv1d(C, dk, kernel_size=K, stride=K, padding=0, bias=False)
        elif convolution_type == 'depthwise':
            self.conv = nn.Conv1d(C, dk, kernel_size=K, stride=K, padding=0, groups=C, bias=False)
            self.conv.weight.data.fill_(1.0)
        elif convolution_type == 'depthwise-separable':
            self.conv = nn.Sequential(
                nn.Conv1d(C, C, kernel_size=K, stride=K, padding=0, groups=C, bias=False),
                nn.Conv1d(C, dk, kernel_size=1, stride=1, padding=0, bias=False))
        # (any other string leaves the module without a conv, as in the reference)

        self._candidate_override: Optional[torch.Tensor] = None
        self.stage_timer = None   # callable(label): records a CUDA event between the stage calls
        self._packed = None
        self._packed_key = None
        self._spatial_cache = {}
        self._calls = _NotCopied()

    # -- host-side helpers --------------------------------------------------------------
    @property
    def candidate_override(self) -> Optional[torch.Tensor]:
        """Fixes the candidate set of the sampled modes (instead of a fresh draw per call)."""
        return self._candidate_override

    @candidate_override.setter
    def candidate_override(self, cand: Optional[torch.Tensor]) -> None:
        if cand is not None:
            ops.check_candidates(cand)      # negatives here; the upper bound once T is known
        self._candidate_override = cand
        self._override_checked_T = None

    def _spec(self) -> LayerSpec:
        return LayerSpec(self.d_hidden, self.num_heads, self.K, self.sampling_type, self.magnitude_type,
                         self.convolution_type, self.softmax_topk_val, self.coordinate_encoding,
                         self.seq_length)

    def _conv_params(self):
        if self.convolution_type == 'depthwise-separable':
            return (self.conv[0].weight, self.conv[1].weight)
        return (self.conv.weight,)

    def _weight_modules(self):
        conv = self.conv if self.convolution_type == 'depthwise-separable' else (self.conv,)
        return (self.W_q, self.W_k, self.W_v, self.W_o, *conv)

    def packed_weights(self, dtype, device):
        params = (self.W_q.weight, self.W_k.weight, self.W_v.weight, self.W_o.weight) + self._conv_params()
        key = (dtype, device) + tuple((p.data_ptr(), p._version) for p in params)
        if self._packed_key != key:
            self._packed = ops.pack_weights(self._spec(), self.W_q.weight, self.W_k.weight, self.W_v.weight,
                                            self.W_o.weight, self._conv_params(), dtype, device)
            self._packed_key = key
        return self._packed

    def candidates(self, T: int, device) -> Optional[torch.Tensor]:
        """Candidate token indices for this call, drawn as the reference draws them
        (layers.py:284, 297) unless ``candidate_override`` is set."""
        if self.sampling_type == 'all':
            return None
        if self._candidate_override is not None:
            if getattr(self, "_override_checked_T", None) != T:
                ops.check_candidates(self._candidate_override, T)    # once per sequence length
                self._override_checked_T = T
            return self._candidate_override.to(device)
        if self.sampling_type == 'random':
            return torch.randperm(T, device=device)[:self.num_samples]
        if self.sampling_type == 'spatial':
            key = (T, str(device))
            kept = self._spatial_cache.get(key)
            if kept is None:
                kept = torch.linspace(0 + self.sample_padding, T - self.sample_padding - 1, self.num_samples,
                                      device=device).long()
                if not capturing(kept.device):
                    self._spatial_cache[key] = kept
            return kept
        raise ValueError("Invalid sampling_type. Must be one of ['all', 'random', 'spatial']")

    def kernel_candidates(self, T: int, device) -> Optional[torch.Tensor]:
        """``candidates`` as the kernels read them (int32), converted by every call on its own stream: a set that is
        changed in place is followed, and a captured graph holds the conversion and its memory.  The set of 'spatial' never
        changes: it is converted once, kept as long as the layer, and complete before any stream can see it."""
        override = self._candidate_override
        cand = self.candidates(T, device if override is None else override.device)
        if cand is None:
            return None
        if cand.device.type == "cpu" and device.type == "cuda":
            return self._device_copy(cand, device)
        key = (T, str(device))
        if cand is not self._spatial_cache.get(key):
            return cand.to(device=device, dtype=torch.int32).contiguous()
        key += (torch.int32,)
        kept = self._spatial_cache.get(key)
        if kept is None:
            kept = cand.to(torch.int32)
            if capturing(kept.device):
                return kept
            if kept.is_cuda:
                torch.cuda.current_stream(kept.device).synchronize()
            self._spatial_cache[key] = kept
        return kept

    def _device_copy(self, cand, device) -> torch.Tensor:
        """A set in host memory on ``device``, copied again when its values change (the copy has arrived when the call
        returns, and cannot be made while a graph is captured).  A copy that a graph was captured with is kept as long as the
        layer."""
        copies = self.__dict__.get("_copies")
        if copies is None:
            copies = self._copies = _NotCopied()
        now = cand.to(torch.int32)
        values, kept = copies.get(device, (None, None))
        if kept is None or not torch.equal(values, now):
            kept = now.to(device)
            copies[device] = (now.clone(), kept)
        if capturing(device):
            copies.setdefault("captured", []).append(kept)
        else:
            kept.record_stream(torch.cuda.current_stream(device))
        return kept

    def candidate_count(self, T: int, device) -> int:
        """S of a call over T tokens (without a draw)."""
        if self.sampling_type == 'random' and self._candidate_override is None:
            return len(range(T)[:self.num_samples])
        if self._candidate_override is not None and self.sampling_type != 'all':
            return self._candidate_override.numel()
        cand = self.candidates(T, device)
        return T if cand is None else cand.numel()

    def _check_mode(self, x):
        if not x.is_cuda:
            raise RuntimeError("convnn_b200.MultiHeadConvNNAttention runs on CUDA (sm_100a) only; "
                               "there is no CPU path")
        if torch.is_grad_enabled() and (x.requires_grad or any(p.requires_grad for p in self.parameters())):
            raise RuntimeError("convnn_b200 is forward-only: call it under torch.no_grad() "
                               "(training / backward is outside this library)")
        if self.training and self.attention_dropout > 0:
            raise RuntimeError("convnn_b200 is forward-only: dropout > 0 needs module.eval()")
        if self.magnitude_type not in ('cosine', 'matmul', 'euclidean'):
            raise ValueError(f"unknown magnitude_type {self.magnitude_type!r}")

    def forward(self, x, out: Optional[torch.Tensor] = None, residual: Optional[torch.Tensor] = None):
        """``layer(x)``; with ``residual`` the caller's skip connection is folded into the last
        store (``residual + layer(x)``), with ``out`` the result is written in place."""
        self._check_mode(x)
        if self.stage_timer is not None or self._packed is None or x.dim() != 3:
            return self._forward_general(x, out, residual)
        key = (x.shape, x.dtype, x.device)
        calls = self.__dict__.get("_calls")
        if calls is None:             # saved as a whole before there were any
            calls = self._calls = _NotCopied()
        call = calls.get(key)
        if call is not None:
            y = call(self, x, out, residual) if call.watch.unchanged(self) else None
            if y is not None:
                return y
            calls.clear()             # those of other shapes hold the same weights as they were
        if capturing(x.device) or not registered(*self._weight_modules()):
            return self._forward_general(x, out, residual)
        if len(calls) >= 16:
            calls.clear()
        call = calls[key] = _LayerCall(self, x)
        y = call(self, x, out, residual)
        return self._forward_general(x, out, residual) if y is None else y

    def _forward_general(self, x, out, residual):
        """The call with nothing prepared for it."""
        B, T, D = x.shape
        cand = self.kernel_candidates(T, x.device)
        packed = self.packed_weights(x.dtype, x.device)
        if self.stage_timer is not None:
            return self._forward_staged(x, packed, cand, out, residual)
        return ops.forward(self._spec(), x, packed, cand, out=out, residual=residual)

    def prenorm_supported(self, x) -> bool:
        """Whether ``forward_prenorm`` takes this input (bfloat16, sampling 'all', a K/V/Q weight tile
        that stays resident in shared memory); otherwise the caller normalises and calls ``forward``."""
        return x.is_cuda and self.prenorm_supported_shape(x.shape[0], x.shape[1], x.dtype)

    def prenorm_supported_shape(self, B: int, T: int, dtype) -> bool:
        """``prenorm_supported`` for a CUDA input (B, T, d_hidden) of ``dtype`` that does not exist yet."""
        return (dtype == torch.bfloat16 and self.stage_timer is None and
                ops.prenorm_forward_supported(self._spec(), B, T, dtype))

    def forward_prenorm(self, x, moments, norm: nn.LayerNorm, residual: Optional[torch.Tensor] = None,
                        want_moments: bool = False, skip_out_proj: bool = False):
        """``layer(norm(x))`` (``+ residual``) from the rows ``x`` BEFORE ``norm`` and their moments,
        the LayerNorm folded into the K/V/Q projection.  Returns (out, moments of out or None).  With
        ``skip_out_proj`` (num_heads = 1) the result is the layer's output BEFORE ``W_o``, for a caller
        that fuses the projection into what follows (``ops.outproj_mlp`` with ``self.packed_w_o``)."""
        self._check_mode(x)
        _, w_conv, w_pw, w_o = self.packed_weights(x.dtype, x.device)
        wf, wx = self.folded_qkv(norm, x.dtype, x.device)
        return ops.prenorm_forward(self._spec(), x, moments, norm.eps, (wf, wx, w_conv, w_pw, None if skip_out_proj else w_o),
                                   residual=residual, want_moments=want_moments)

    @property
    def packed_w_o(self):
        """The output projection as last packed."""
        return self._packed[3]

    def folded_qkv(self, norm: nn.LayerNorm, dtype, device):
        """The packed K/V/Q weight with ``norm`` folded in (``ops.fold_layernorm``)."""
        w_qkv = self.packed_weights(dtype, device)[0]
        if getattr(self, "_folded", None) is None:
            self._folded = _PackedParams()
        return self._folded.get((w_qkv, norm.weight, norm.bias), dtype, device, lambda: ops.fold_layernorm(
            w_qkv.view(-1, w_qkv.shape[-1]), None, norm.weight.detach().to(device, dtype),
            norm.bias.detach().to(device, dtype)))

    def _forward_staged(self, x, packed, cand, out, residual=None):
        """The same kernels in the same order as ``convnn_b200_forward``, issued through the
        four stage entry points so a profiler hook can bracket each with CUDA events."""
        spec, mark = self._spec(), self.stage_timer
        w_qkv, w_conv, w_pw, w_o = packed
        mark("begin")
        q, k, v, qs, ks = ops.qkv_proj(spec, x, w_qkv, cand)
        mark("qkv_proj")
        idx, val = ops.sim_topk(spec, q, k, qs, ks, cand)
        mark("sim_topk")
        o = ops.gather_conv(spec, v, idx, val, w_conv, w_pw, S=q.shape[1])
        mark("gather_conv")
        y = ops.out_proj(spec, o, w_o, out=out, S=q.shape[1], residual=residual)
        mark("out_proj")
        return y


def _library_call(x: torch.Tensor, what: str) -> None:
    if not x.is_cuda:
        raise RuntimeError(f"convnn_b200.{what} runs on CUDA (sm_100a) only; there is no CPU path")
    if torch.is_grad_enabled() and x.requires_grad:
        raise RuntimeError("convnn_b200 is forward-only: call it under torch.no_grad() "
                           "(training / backward is outside this library)")


class _PackedParams:
    """Kernel-side copies of a module's parameters, rebuilt when a parameter changes."""

    def __init__(self):
        self._key, self._val = None, None

    def get(self, params, dtype, device, build):
        key = (dtype, device) + tuple((p.data_ptr(), p._version) for p in params)
        if key != self._key:
            self._val, self._key = build(), key
        return self._val


class MultiHeadAttention(WatchedModule):
    """Softmax attention half of MultiHeadBranchingAttention (reference layers.py:90-130):
    bias-free W_q/W_k/W_v/W_o, softmax(QK^T / sqrt(d_k)) V.  The modules hold the parameters (same
    ``state_dict`` keys as the reference); the forward runs in libconvnn_b200: one packed
    three-output projection, the softmax-attention kernel, the output projection."""

    def __init__(self, d_hidden, num_heads, attention_dropout):
        super().__init__()
        assert d_hidden % num_heads == 0, "d_hidden must be divisible by num_heads"
        self.d_hidden, self.num_heads, self.d_k = d_hidden, num_heads, d_hidden // num_heads
        self.dropout = nn.Dropout(attention_dropout)
        self.W_q = nn.Linear(d_hidden, d_hidden, bias=False)
        self.W_k = nn.Linear(d_hidden, d_hidden, bias=False)
        self.W_v = nn.Linear(d_hidden, d_hidden, bias=False)
        self.W_o = nn.Linear(d_hidden, d_hidden, bias=False)
        self._packed = _PackedParams()

    def _weight_modules(self):
        return self.W_q, self.W_k, self.W_v, self.W_o

    def packed_weights(self, dtype, device):
        params = (self.W_q.weight, self.W_k.weight, self.W_v.weight, self.W_o.weight)
        return self._packed.get(params, dtype, device, lambda: (
            torch.stack([p.detach().to(device, dtype) for p in params[:3]]).contiguous(),
            self.W_o.weight.detach().to(device, dtype).contiguous()))

    def forward(self, x, mask=None, out: Optional[torch.Tensor] = None):
        _library_call(x, "MultiHeadAttention")
        if mask is not None:
            raise RuntimeError("convnn_b200.MultiHeadAttention takes no mask (the reference's ViT never passes one)")
        if self.training and self.dropout.p > 0:
            raise RuntimeError("convnn_b200 is forward-only: dropout > 0 needs module.eval()")
        w_qkv, w_o = self.packed_weights(x.dtype, x.device)
        return ops.softmax_attention(x, w_qkv, w_o, self.num_heads, out=out)


class MultiHeadConv1dAttention(WatchedModule):
    """Conv1d half of MultiHeadBranchingConv (reference layers.py:452-500): Linear, per-head
    Conv1d(d_k, d_k, kernel_size, padding='same'), the reference's flat head reinterpretation,
    Linear.  Parameters as in the reference; the forward runs in libconvnn_b200."""

    def __init__(self, d_hidden, num_heads, kernel_size):
        super().__init__()
        assert d_hidden % num_heads == 0, "d_hidden must be divisible by num_heads"
        self.d_hidden, self.num_heads, self.d_k = d_hidden, num_heads, d_hidden // num_heads
        self.kernel_size, self.stride = kernel_size, 1
        self.W_x = nn.Linear(d_hidden, d_hidden)
        self.W_o = nn.Linear(d_hidden, d_hidden)
        self.in_channels = self.out_channels = self.d_k
        self.conv = nn.Conv1d(self.d_k, self.d_k, kernel_size=kernel_size, stride=1, padding="same")
        self._packed = _PackedParams()

    def _weight_modules(self):
        return self.W_x, self.conv, self.W_o

    def packed_weights(self, dtype, device):
        params = (self.W_x.weight, self.W_x.bias, self.conv.weight, self.conv.bias, self.W_o.weight, self.W_o.bias)

        def build():
            cvt = lambda t: t.detach().to(device, dtype).contiguous()
            # (d_k out, d_k in, kernel_size) -> (d_k out, kernel_size, d_k in): a (d_k, kernel_size * d_k) matrix
            return (cvt(self.W_x.weight), cvt(self.W_x.bias), cvt(self.conv.weight.permute(0, 2, 1)),
                    cvt(self.conv.bias), cvt(self.W_o.weight), cvt(self.W_o.bias))
        return self._packed.get(params, dtype, device, build)

    def forward(self, x, out: Optional[torch.Tensor] = None):
        _library_call(x, "MultiHeadConv1dAttention")
        w_x, b_x, w_c, b_c, w_o, b_o = self.packed_weights(x.dtype, x.device)
        return ops.conv1d_attention(x, w_x, b_x, w_c, b_c, w_o, b_o, self.num_heads, self.kernel_size, out=out)


class _Branching(WatchedModule):
    def _init_common(self, d_hidden, num_heads, attention_dropout, K, sampling_type, num_samples,
                     sample_padding, magnitude_type, seq_length, coordinate_encoding, convolution_type,
                     softmax_topk_val, branch_ratio):
        self.d_hidden = d_hidden
        self.num_heads = num_heads
        self.attention_dropout = attention_dropout
        self.K = K
        self.sampling_type = sampling_type
        self.num_samples = int(num_samples)
        self.sample_padding = int(sample_padding) if sampling_type == 'spatial' else 0
        self.magnitude_type = magnitude_type
        self.seq_length = seq_length
        self.coordinate_encoding = coordinate_encoding
        self.branch_ratio = branch_ratio
        self.d_hidden_convnn = int(branch_ratio * d_hidden)
        if branch_ratio != 0:
            self.convnn = MultiHeadConvNNAttention(
                d_hidden=self.d_hidden_convnn, num_heads=num_heads, attention_dropout=attention_dropout, K=K,
                sampling_type=sampling_type, num_samples=num_samples, sample_padding=sample_padding,
                magnitude_type=magnitude_type, seq_length=seq_length, coordinate_encoding=coordinate_encoding,
                convolution_type=convolution_type, softmax_topk_val=softmax_topk_val)

    def _two_branches(self, x, other, residual=None):
        """Both branches read their channel slice of x in place and write their slice of the
        concat buffer in place (no slice copy in, no cat copy out); then pointwise_linear with
        its bias, and the caller's skip connection if given, folded into one GEMM epilogue
        (reference layers.py:574-577, 648-651; vit.py:264)."""
        dc = self.d_hidden_convnn
        cat = torch.empty(x.shape, dtype=x.dtype, device=x.device)
        self.convnn(x[:, :, :dc], out=cat[:, :, :dc])
        other(x[:, :, dc:], out=cat[:, :, dc:])
        pw = self.pointwise_linear
        return ops.linear(cat, pw.weight, pw.bias, residual=residual)


class MultiHeadBranchingAttention(_Branching):
    def __init__(self, d_hidden, num_heads, attention_dropout, K, sampling_type, num_samples, sample_padding,
                 magnitude_type, seq_length=197, coordinate_encoding=False, convolution_type='depthwise',
                 softmax_topk_val=True, branch_ratio=0.5):
        super().__init__()
        self._init_common(d_hidden, num_heads, attention_dropout, K, sampling_type, num_samples, sample_padding,
                          magnitude_type, seq_length, coordinate_encoding, convolution_type, softmax_topk_val,
                          branch_ratio)
        self.d_hidden_attention = d_hidden - self.d_hidden_convnn
        if branch_ratio != 1:
            self.attention = MultiHeadAttention(self.d_hidden_attention, num_heads, attention_dropout)
        self.pointwise_linear = nn.Linear(d_hidden, d_hidden)

    def forward(self, x, residual: Optional[torch.Tensor] = None):
        # The reference swaps the degenerate cases (ratio 0 calls the ConvNN branch that was
        # not built and vice versa, layers.py:643-646) and fails with AttributeError; so do we.
        if self.branch_ratio == 0:
            y = self.convnn(x)
        elif self.branch_ratio == 1:
            y = self.attention(x)
        else:
            return self._two_branches(x, self.attention, residual)
        return y if residual is None else residual + y


class MultiHeadBranchingConv(_Branching):
    def __init__(self, d_hidden, num_heads, attention_dropout, kernel_size, K, sampling_type, num_samples,
                 sample_padding, magnitude_type, seq_length=197, coordinate_encoding=False,
                 convolution_type='depthwise', softmax_topk_val=True, branch_ratio=0.5):
        super().__init__()
        self.kernel_size = kernel_size
        self._init_common(d_hidden, num_heads, attention_dropout, K, sampling_type, num_samples, sample_padding,
                          magnitude_type, seq_length, coordinate_encoding, convolution_type, softmax_topk_val,
                          branch_ratio)
        self.d_hidden_conv1d = d_hidden - self.d_hidden_convnn
        if branch_ratio != 1:
            self.conv1d = MultiHeadConv1dAttention(self.d_hidden_conv1d, num_heads, kernel_size)
        self.pointwise_linear = nn.Linear(d_hidden, d_hidden)

    def forward(self, x, residual: Optional[torch.Tensor] = None):
        if self.branch_ratio == 0:
            y = self.conv1d(x)
        elif self.branch_ratio == 1:
            y = self.convnn(x)
        else:
            return self._two_branches(x, self.conv1d, residual)
        return y if residual is None else residual + y
