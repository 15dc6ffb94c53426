"""The single-token step of a GPT-2 model as one kernel launch (fa_b200_gpt_step).

A `StepPlan` is what the launch needs of a model: the table of its parameters' addresses on the GPU
and, per stream, a workspace.  gpt2.GPTModel makes one in prepare_for_inference() and uses it for
every forward of one token per sequence against K/V caches that the kernel can take; other shapes
go layer by layer.
"""
from __future__ import annotations

import ctypes
import operator
import weakref
from collections import OrderedDict

import torch
import torch.nn as nn

from . import _lib

MAX_BATCH = 8
MAX_PAIRS = 256            # sequences x heads
MAX_LAYERS = 64
MAX_WIDTH = 1600
MAX_VOCAB = 1 << 24        # fewer than that
MAX_CACHE_ROWS = 1 << 22
MAX_STRIDE = (1 << 31) - 1    # of a cache's rows and heads
PLAIN_TENSORS = (torch.Tensor, nn.Parameter)     # a subclass may keep its numbers in another form
MAX_WORKSPACES = 8         # streams that keep a workspace (about 1 MB each)


_workspaces = weakref.WeakValueDictionary()     # every workspace that is still somebody's


def clear_workspaces(device):
    """Zero the workspaces on a device, after a kernel gave up a wait: it may have left counters in them that
    the next launch would count on from."""
    torch.cuda.synchronize(device)
    for ws in list(_workspaces.values()):
        if ws.device == device:
            ws.zero_()
    torch.cuda.synchronize(device)


class ModelWatch:
    """The modules, parameters and settings of a GPTModel that the paths past its modules stand in for (the
    one-launch step here, the binding's loop over the blocks of a prompt), as they are when this is made.
    `holds()` says whether the model still consists of the same ones; it runs on every call, so it is
    a comparison of identities without a loop in Python (37 entries a block: 17 us for GPT-2 small)."""

    UNREAD = ("W_query", "W_key", "W_value", "dropout", "drop_shortcut")    # replaced by _qkv_w / identities

    def __init__(self, model):
        entries = []                   # (dict, key, value): parameters, submodules, plain attributes
        tensors = []
        todo = [model]
        while todo:
            m = todo.pop()
            d = m.__dict__
            for name, t in m._parameters.items():
                entries.append((m._parameters, name, t))
                if t is not None:
                    tensors.append(t)
            for name, child in m._modules.items():
                if name not in self.UNREAD:
                    entries.append((m._modules, name, child))
                    if child is not None:
                        todo.append(child)
            entries += [(d, name, d[name]) for name in ("impl_type", "num_heads", "d_out", "eps", "_qkv_w", "_qkv_b") if name in d]
        called = called_modules(model)
        entries += [(m.__dict__, "forward", m.__dict__.get("forward")) for m in called]
        self.hooks = [d for m in called for d in (m._forward_hooks, m._forward_pre_hooks)]
        self.hooks += [nn.modules.module._global_forward_hooks, nn.modules.module._global_forward_pre_hooks]
        self.dicts, self.keys, self.values = (list(part) for part in zip(*entries))
        self.tensors, self.addresses = tensors, [t.data_ptr() for t in tensors]
        self.top = model._modules           # (a shallow copy of a model has its own)
        self.blocks = model.trf_blocks._modules
        self.n_blocks = len(self.blocks)

    def hooked(self):
        """Whether somebody wants to hear of a call that those paths do not make."""
        return any(self.hooks)

    def holds(self, model):
        return (self.top is model._modules and all(map(operator.is_, map(dict.get, self.dicts, self.keys), self.values))
                and len(self.blocks) == self.n_blocks
                and list(map(torch.Tensor.data_ptr, self.tensors)) == self.addresses)


def called_modules(model):
    """The modules that the prepared model's own loops call (of the others they read the parameters)."""
    called = [model.tok_emb, model.pos_emb, model.drop_emb]
    for blk in model.trf_blocks:
        att, ff = getattr(blk, "att", None), getattr(blk, "ff", None)
        layers = getattr(ff, "layers", None)
        called += [att, ff, getattr(att, "out_proj", None), layers[2] if isinstance(layers, nn.Sequential) and len(layers) > 2 else None]
    return [m for m in called if isinstance(m, nn.Module)]


def plain_modules(model):
    """Whether the model is built of the modules that those paths know, one head size and width throughout."""
    from . import gpt2
    cfg = model.cfg
    width, heads = cfg["emb_dim"], cfg["n_heads"]
    if type(model.final_norm) is not gpt2.LayerNorm or type(model.out_head) is not nn.Linear:
        return False
    if type(model.tok_emb) is not nn.Embedding or type(model.pos_emb) is not nn.Embedding:
        return False
    for blk in model.trf_blocks:
        if type(blk) is not gpt2.TransformerBlock or type(blk.att) is not gpt2.MultiHeadAttention or type(blk.ff) is not gpt2.FeedForward:
            return False
        att, layers = blk.att, blk.ff.layers
        if type(blk.norm1) is not gpt2.LayerNorm or type(blk.norm2) is not gpt2.LayerNorm or type(layers) is not nn.Sequential:
            return False
        if type(att.out_proj) is not nn.Linear or type(layers[0]) is not nn.Linear or type(layers[2]) is not nn.Linear:
            return False
        if att.num_heads != heads or att.d_out != width or att.impl_type != "cuda" or att._qkv_w is None:
            return False
        if blk.norm1.eps != model.final_norm.eps or blk.norm2.eps != model.final_norm.eps:
            return False
    return not any("forward" in m.__dict__ for m in called_modules(model))


class StepPlan:
    """Parameter table of one prepared bf16 model.  `make` returns None for a model the kernel does
    not take."""

    @classmethod
    def make(cls, model):
        cfg = model.cfg
        width, heads, layers = cfg["emb_dim"], cfg["n_heads"], len(model.trf_blocks)
        if width != 64 * heads or width > MAX_WIDTH or not 1 <= layers <= MAX_LAYERS or heads > MAX_PAIRS:
            return None
        if not plain_modules(model):
            return None
        plan = cls()
        plan.device = model.tok_emb.weight.device
        plan.weights = []    # what the table points at
        rows = []

        def take(module, name, shape, optional=False):
            return plan._take(module._parameters.get(name), shape, optional)

        try:
            for blk in model.trf_blocks:
                att, fc, out = blk.att, blk.ff.layers[0], blk.ff.layers[2]
                rows.append([take(blk.norm1, "scale", (width,)), take(blk.norm1, "shift", (width,)),
                             plan._take(att._qkv_w, (3 * width, width)), plan._take(att._qkv_b, (3 * width,), optional=True),
                             take(att.out_proj, "weight", (width, width)), take(att.out_proj, "bias", (width,)),
                             take(blk.norm2, "scale", (width,)), take(blk.norm2, "shift", (width,)),
                             take(fc, "weight", (4 * width, width)), take(fc, "bias", (4 * width,)),
                             take(out, "weight", (width, 4 * width)), take(out, "bias", (width,))])
            plan.vocab = model.out_head.weight.shape[0]
            plan.positions = model.pos_emb.weight.shape[0]
            if plan.vocab >= MAX_VOCAB:
                return None
            plan.ends = [take(model.tok_emb, "weight", (plan.vocab, width)),
                         take(model.pos_emb, "weight", (plan.positions, width)),
                         take(model.final_norm, "scale", (width,)), take(model.final_norm, "shift", (width,)),
                         take(model.out_head, "weight", (plan.vocab, width))]
        except TypeError:
            return None
        plan.qkv = [(blk.att, blk.att._qkv_w, blk.att._qkv_b) for blk in model.trf_blocks]
        plan.heads, plan.layers, plan.eps = heads, layers, model.final_norm.eps
        plan.table = torch.tensor(rows, dtype=torch.int64).to(plan.device)
        plan.recorded = model.__dict__.setdefault("_recorded_tables", [])
        plan.workspaces = OrderedDict()
        return plan

    def _take(self, t, shape, optional=False):
        """The address of a parameter of this shape (0 for one that is not there and need not be)."""
        if t is None and optional:
            return 0
        if (type(t) not in PLAIN_TENSORS or not t.is_cuda or t.device != self.device or t.dtype != torch.bfloat16 or tuple(t.shape) != shape
                or not t.is_contiguous() or t.data_ptr() % 16):
            raise TypeError("not a dense bf16 CUDA parameter of the expected shape")
        self.weights.append(t)
        return t.data_ptr()

    def memory(self):
        """Everything a launch reads through this plan: the table and the tensors whose addresses are in
        it, under names of their own (a parameter that is moved or replaced takes its storage along).  For
        a recorded launch, which reads them for as long as it is replayed."""
        return [t.detach() for t in [self.table] + self.weights]

    def _caches(self, kv_caches, batch):
        """The caches' addresses and common shape, or None when the kernel cannot take them."""
        if len(kv_caches) != self.layers:
            return None
        k0 = kv_caches[0][0]
        shape, stride = k0.shape, k0.stride()
        if (k0.dim() != 4 or shape[0] != batch or shape[2] != self.heads or shape[3] != 64 or stride[3] != 1
                or k0.device != self.device):
            return None
        table = (ctypes.c_void_p * (2 * self.layers))()
        for i, pair in enumerate(kv_caches):
            for j in (0, 1):
                t = pair[j]
                if t.dtype != torch.bfloat16 or t.shape != shape or t.stride() != stride or not t.is_cuda:
                    return None
                table[j * self.layers + i] = t.data_ptr()
        if any(s % 8 for s in stride[:3]) or any(s <= 0 for s in stride[:3]):
            return None
        if shape[1] > MAX_CACHE_ROWS or max(stride[1], stride[2]) > MAX_STRIDE:
            return None
        return table, shape[1], stride

    def new_workspace(self, batch):
        """A zeroed workspace, or None for a batch that the kernel does not take."""
        need = _lib.load().fa_b200_gpt_step_workspace_bytes(batch, self.heads)
        if need <= 0:
            return None
        ws = torch.zeros(need, dtype=torch.uint8, device=self.device)
        _workspaces[id(ws)] = ws
        return ws

    def _workspace(self, batch, stream):
        """A zeroed workspace that only this stream uses (a launch leaves its counters at zero)."""
        if torch.cuda.is_current_stream_capturing():
            # The graph is the caller's: it reads the table for as long as it is replayed, so the model keeps
            # it (a few KB).  Weights that are replaced meanwhile are the caller's business as ever, but no
            # address that the kernel follows becomes something else.
            if not any(t is self.table for t in self.recorded):
                self.recorded.append(self.table)
            return self.new_workspace(batch)     # belongs to the graph
        key = (stream, batch)
        ws = self.workspaces.get(key)
        if ws is None:
            ws = self.workspaces[key] = self.new_workspace(batch)
            while len(self.workspaces) > MAX_WORKSPACES:
                self.workspaces.popitem(last=False)
        return ws

    def step(self, ids, kv_caches, pos, advance=False, next_ids=None, workspace=None):
        """Logits [B, 1, vocab] of one new token per sequence, or None when this call is not one for
        the kernel.  `ids` int64 [B, 1]; `pos` an int or a gpt2.DevicePosition (which `advance`
        moves on); `next_ids` int64 [B] (any stride) receives the argmax of each row."""
        batch = ids.shape[0]
        if not 1 <= batch <= MAX_BATCH or batch * self.heads > MAX_PAIRS or ids.device != self.device:
            return None
        found = self._caches(kv_caches, batch)
        if found is None:
            return None
        table, rows, stride = found
        on_device = hasattr(pos, "index") and hasattr(pos, "length")
        if not on_device:
            if isinstance(pos, torch.Tensor) or not hasattr(pos, "__index__"):
                return None
            pos = operator.index(pos)            # (numpy's integers, too)
            if not 0 <= pos < min(rows, self.positions):
                return None
        if ids.dtype != torch.int64:
            ids = ids.long()
        stream = torch.cuda.current_stream(self.device).cuda_stream
        ws = self._workspace(batch, stream) if workspace is None else workspace
        logits = torch.empty(batch, 1, self.vocab, dtype=torch.bfloat16, device=self.device)
        p = _lib.FaGptStepParams()
        p.layers = self.table.data_ptr()
        p.tok_emb, p.pos_emb, p.lnf_scale, p.lnf_shift, p.head_w = self.ends
        p.ids, p.ids_stride = ids.data_ptr(), ids.stride(0)
        if on_device:
            p.pos_device, p.length_device = pos.index.data_ptr(), pos.length.data_ptr()
        else:
            p.pos = pos
        p.advance = 1 if advance else 0
        p.k_cache = ctypes.addressof(table)
        p.v_cache = ctypes.addressof(table) + 8 * self.layers
        p.cache_strides[0], p.cache_strides[1], p.cache_strides[2] = stride[0], stride[1], stride[2]
        if batch == 1:
            p.cache_strides[0] = 64              # never used to address anything
        p.logits = logits.data_ptr()
        if next_ids is not None:
            p.next_ids, p.next_stride = next_ids.data_ptr(), next_ids.stride(0)
        p.workspace, p.workspace_bytes = ws.data_ptr(), ws.numel()
        p.n_layers, p.B, p.H, p.vocab = self.layers, batch, self.heads, self.vocab
        p.cache_rows, p.n_positions, p.eps = rows, self.positions, self.eps
        p.device, p.stream = self.device.index, stream
        rc = _lib.load().fa_b200_gpt_step(ctypes.byref(p))
        if rc != 0:
            raise RuntimeError(f"generation step failed ({rc}): {_lib.strerror(rc)}")
        return logits
