"""Host plan of a ViT forward: everything ``convnn_b200_model_forward`` reads, prepared once.

A ViT-Tiny forward is 64 launches; issued one binding call at a time they cost the host 1.14 ms (measured, one
image), most of it argument handling and shape logic between the calls, so batches below ~100 images ran at the
host's pace.  A plan holds the model's weight pointers, packed copies, layer descriptors and workspace size for
one input shape; a forward then is a validity check, two allocations and one native call.  Candidate sets are not
part of it but taken from the layers on every call: a captured graph would read a plan's copy after the plan is gone.

A plan is used only while it describes the model: ``Watch.unchanged()`` compares the attribute stamps of this package's
modules, the module tree, and identity, version counter and address of every parameter and buffer, ``Plan.unchanged()``
also the numbers read from other objects (``eps`` of the norms, the patch size), and a call that finds a difference builds
a new plan.  Anything a plan does not cover (training mode, hooks, a stage timer,
parameters of another dtype or device) takes the op-by-op path in ``vit.py``.
"""
from __future__ import annotations

import ctypes
import threading
import weakref
from collections import OrderedDict

import torch
from torch.nn.modules import module as _nn_module

from . import _capi, layers, ops
from .layers import (MultiHeadAttention, MultiHeadBranchingAttention, MultiHeadBranchingConv, MultiHeadConv1dAttention,
                     MultiHeadConvNNAttention, Watch, registered)

MAX_PLANS = 32                      # input shapes remembered per model, the latest used ones (host memory only)
_SEEN = object()                    # a shape that has been called once
_plans: "weakref.WeakKeyDictionary" = weakref.WeakKeyDictionary()
_lock = threading.Lock()            # the order of a model's entries


def _remember(per_model, key, entry):
    with _lock:
        per_model[key] = entry
        per_model.move_to_end(key)
        while len(per_model) > MAX_PLANS:
            per_model.popitem(last=False)


class Plan:
    def __init__(self, model, x: torch.Tensor, act: torch.dtype, watch: Watch):
        a = model.args
        B, C, Hh, Ww = x.shape
        T, D = model.n_patches + 1, model.d_hidden
        self.watch = watch
        self.keep = []              # tensors whose addresses the structs hold
        self.read = []              # (object, attribute, value) of what the structs hold of objects outside this package
        self.sampled = []           # (block index, attention layer, candidates the plan was made for)
        blocks = list(model.transformer_encoder)
        self.blocks = (_capi.ConvnnBlock * max(1, len(blocks)))()
        for i, blk in enumerate(blocks):
            self._block(i, blk, B, T, D, act, x.device)
        pe, pemb, cls = model.positional_encoding, model.patch_embedding, model.positional_encoding.cls_tokens
        conv = pemb.linear_projection
        m = self.model = _capi.ConvnnModel()
        m.dtype, m.B, m.T, m.D = ops._dtype_code(act), B, T, D
        m.n_blocks, m.classes = len(blocks), model.classifier.weight.shape[0]
        m.channels, m.height, m.width, m.patch = C, Hh, Ww, self._attr(a, "patch_size")
        m.embed_eps = self._attr(pemb.norm, "eps")
        m.blocks = ctypes.cast(self.blocks, ctypes.POINTER(_capi.ConvnnBlock))
        m.patch_w, m.patch_b = self._ptr(conv.weight.view(D, -1)), self._ptr(conv.bias)
        m.embed_norm_w, m.embed_norm_b = self._ptr(pemb.norm.weight), self._ptr(pemb.norm.bias)
        m.cls, m.pe = self._ptr(cls.view(-1)), self._ptr(pe.pe.view(-1, D)[:T])
        m.head_w, m.head_b = self._ptr(model.classifier.weight), self._ptr(model.classifier.bias)
        m.images_u8, self.mean = int(x.dtype == torch.uint8), None
        if m.images_u8:
            _, mean, inv_std = model.pixel_stats(x.device)
            self.mean = mean
            m.pixel_mean, m.pixel_inv_std = self._ptr(mean), self._ptr(inv_std)
        self.act, self.out_shape, self.lock = act, (B, m.classes), threading.Lock()
        L = _capi.lib()
        self.call, self.arg = L.convnn_b200_model_forward, ctypes.byref(m)
        self.workspace_bytes = L.convnn_b200_model_workspace_bytes(self.arg)
        self.least_bytes = L.convnn_b200_model_workspace_least_bytes(self.arg)

    def unchanged(self, model) -> bool:
        return (self.watch.unchanged(model) and not any(self.watch.hooks) and
                all([getattr(o, name) == value for o, name, value in self.read]))

    # -- construction -------------------------------------------------------------------------------
    def _attr(self, o, name):
        value = getattr(o, name)
        self.read.append((o, name, value))
        return value

    def _ptr(self, t):
        if t is None:
            return None
        if not t.is_contiguous():
            t = t.contiguous()
        self.keep.append(t)
        return t.data_ptr()

    def _folded(self, b, names, fold):
        wf, wx = fold
        setattr(b, names[0], self._ptr(wf))
        setattr(b, names[1], self._ptr(wx))

    def _layer(self, b, i, att, B, T, act, device):
        """The ConvNN layer of a block: descriptor, packed weights."""
        S = att.candidate_count(T, device)
        if att.sampling_type != "all":
            self.sampled.append((i, att, S))
        b.layer = ops.descriptor(att._spec(), B, T, S, act)
        w_qkv, w_conv, w_pw, w_o = att.packed_weights(act, device)
        b.w_qkv, b.w_conv, b.w_pw, b.w_o = (self._ptr(w) for w in (w_qkv, w_conv, w_pw, w_o))

    def _block(self, i, blk, B, T, D, act, device):
        b, att = self.blocks[i], blk.attention
        n1, n2, fc1, fc2 = blk.norm1, blk.norm2, blk.mlp[0], blk.mlp[3]
        branching = isinstance(att, (MultiHeadBranchingAttention, MultiHeadBranchingConv))
        self._layer(b, i, att.convnn if branching else att, B, T, act, device)
        b.d_mlp, b.eps1, b.eps2 = fc1.weight.shape[0], self._attr(n1, "eps"), self._attr(n2, "eps")
        b.norm1_w, b.norm1_b, b.norm2_w, b.norm2_b = (self._ptr(t) for t in (n1.weight, n1.bias, n2.weight, n2.bias))
        b.fc1_w, b.fc1_b, b.fc2_w, b.fc2_b = (self._ptr(t) for t in (fc1.weight, fc1.bias, fc2.weight, fc2.bias))
        if not branching and blk.folds_norm1_shape(B, T, act):
            self._folded(b, ("w_qkv_folded", "w_qkv_extra"), att.folded_qkv(n1, act, device))
        if (blk.fold_layernorm and act == torch.bfloat16 and
                ops.prenorm_linear_supported(*fc1.weight.shape, True)):
            self._folded(b, ("fc1_folded", "fc1_extra"), blk.folded_fc1(act, device))
        b.fuse_mlp = int(blk.fuse_mlp)
        if branching:
            other = att.attention if isinstance(att, MultiHeadBranchingAttention) else att.conv1d
            packed = [self._ptr(w) for w in other.packed_weights(act, device)]
            if isinstance(att, MultiHeadBranchingAttention):
                b.kind, (b.branch_w_in, b.branch_w_out) = _capi.BLOCK_BRANCH_ATTENTION, packed
            else:
                b.kind, b.kernel_size = _capi.BLOCK_BRANCH_CONV1D, other.kernel_size
                (b.branch_w_in, b.branch_b_in, b.branch_w_conv, b.branch_b_conv, b.branch_w_out, b.branch_b_out) = packed
            b.pointwise_w, b.pointwise_b = self._ptr(att.pointwise_linear.weight), self._ptr(att.pointwise_linear.bias)

    # -- a forward ----------------------------------------------------------------------------------
    def _candidates(self, device):
        """This call's candidate sets, one per sampled layer in the order of the layers (a set that several layers share
        is converted once); None: one has another size now."""
        shared, sets = {}, []
        for _, att, S in self.sampled:
            override = att.candidate_override
            cand = None if override is None else shared.get(id(override))
            if cand is None:
                cand = att.kernel_candidates(self.model.T, device)
                shared[id(override)] = cand
            if cand.numel() != S:
                return None
            sets.append(cand)
        return sets

    def run(self, model, x: torch.Tensor):
        """The logits; None where the plan does not describe the call any more."""
        if self.mean is not None and model.pixel_stats(x.device)[1] is not self.mean:
            return None
        if not x.is_contiguous():
            x = x.contiguous()
        dev = x.device
        out = torch.empty(self.out_shape, dtype=self.act, device=dev)
        try:
            ws = torch.empty(self.workspace_bytes, dtype=torch.uint8, device=dev)
        except torch.cuda.OutOfMemoryError:
            # room for one half of a branching block at a time is enough: they run in turn then
            if self.workspace_bytes <= self.least_bytes:
                raise
            self.workspace_bytes = self.least_bytes
            ws = torch.empty(self.least_bytes, dtype=torch.uint8, device=dev)
        args = (self.arg, x.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(), ops._stream(x))
        if self.sampled:
            sets = self._candidates(dev)
            if sets is None:
                return None
            with self.lock:          # the structs are this call's until it returns
                for (i, _, _), cand in zip(self.sampled, sets):
                    self.blocks[i].cand = cand.data_ptr()
                rc = self.call(*args)
        else:
            rc = self.call(*args)
        if rc:
            _capi.check(rc)
        return out


class _Refused:
    """A shape no plan covers, remembered until an attribute of the model or its hooks change."""

    def __init__(self, watch: Watch):
        self.watch, self.hooked = watch, any(watch.hooks)

    def unchanged(self, model) -> bool:
        return self.watch.options_unchanged(model) and any(self.watch.hooks) == self.hooked


def _own(m, cls) -> bool:
    return type(m) is cls and "forward" not in m.__dict__


def _own_attention(att) -> bool:
    """Whether calling the module would run this package's code, on registered weights."""
    if _own(att, MultiHeadConvNNAttention):
        return registered(*att._weight_modules())
    if _own(att, MultiHeadBranchingAttention):
        halves = ("convnn", MultiHeadConvNNAttention), ("attention", MultiHeadAttention)
    elif _own(att, MultiHeadBranchingConv):
        halves = ("convnn", MultiHeadConvNNAttention), ("conv1d", MultiHeadConv1dAttention)
    else:
        return False
    return (0 < att.branch_ratio < 1 and registered(att.pointwise_linear) and
            all(_own(getattr(att, name), cls) and registered(*getattr(att, name)._weight_modules()) for name, cls in halves))


def _covered(model, x: torch.Tensor, act: torch.dtype, watch: Watch) -> bool:
    """Whether a plan can describe this call."""
    from .vit import TransformerEncoder, ViT
    if (type(model) is not ViT or x.dim() != 4 or x.shape[0] < 1 or act not in (torch.float32, torch.bfloat16) or
            tuple(x.shape[1:]) != tuple(model.args.img_size) or not all(type(b) is TransformerEncoder
                                                                        for b in model.transformer_encoder)):
        return False
    if any(watch.hooks):
        return False
    for m in [model] + watch.mods:
        if isinstance(m, layers.WatchedModule) and (m.training or getattr(m, "stage_timer", None) is not None):
            return False
    pe, pemb = model.positional_encoding, model.patch_embedding
    if ("cls_tokens" not in pe._parameters or "pe" not in pe._buffers or
            not registered(pemb.linear_projection, pemb.norm, model.classifier)):
        return False
    for blk in model.transformer_encoder:
        if blk.fuse_out_proj or not _own_attention(blk.attention):
            return False
        if not registered(blk.norm1, blk.norm2, blk.mlp[0], blk.mlp[3]):
            return False
    dev = x.device
    return all([t.dtype == act and t.device == dev and t.is_contiguous() for t in watch.tensors])


def run(model, x: torch.Tensor):
    """The logits through a plan, or None where the op-by-op path has to be taken."""
    per_model = _plans.get(model)
    if per_model is None:
        per_model = _plans.setdefault(model, OrderedDict())
    if _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return None
    key = (x.shape, x.dtype, x.device)
    plan = per_model.get(key)
    if plan is not None and plan is not _SEEN:
        if plan.unchanged(model):
            y = plan.run(model, x) if type(plan) is Plan else None
            if y is not None or type(plan) is not Plan:
                _remember(per_model, key, plan)
                return y
        with _lock:
            per_model.clear()           # those of other shapes hold the same weights as they were
        plan = None
    if layers.capturing(x.device):
        return None
    # The first call of a shape, and the first after a change of the model, goes op by op: it packs weights while
    # the GPU works, and a shape that never returns pays for no plan.  The second call builds the plan.
    if plan is not _SEEN:
        _remember(per_model, key, _SEEN)
        return None
    act = model.patch_embedding.linear_projection.weight.dtype if x.dtype == torch.uint8 else x.dtype
    watch = Watch(model)
    if not _covered(model, x, act, watch):
        _remember(per_model, key, _Refused(watch))
        return None
    plan = Plan(model, x, act, watch)
    if plan.workspace_bytes == 0:           # a shape the library refuses: the op-by-op path raises its error
        return None
    y = plan.run(model, x)
    if y is not None:
        _remember(per_model, key, plan)
    return y
