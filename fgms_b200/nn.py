"""Autograd wrapper around the operator: what dgSPARSE-Lib (the caller named by the reference's README)
puts on top of ``FGMS.backend``.

``sparse_conv(feats, weight, kmap)`` is differentiable in ``feats`` and ``weight``; forward is
``fgms_fusion_fwd_cuda``, backward is ``fgms_bwd_cuda`` (dgrad + wgrad).  ``SparseConv3d`` is the
``nn.Module`` that owns the ``[k_vol, c_in, c_out]`` weight.  Kernel maps are passed in (a
:class:`fgms_b200.gpu_maps.DeviceKernelMap`, or anything with ``kpos / imap / omap / n_in / n_out``
device tensors): layers at one resolution share one map, which is the map caching the reference's driver
does by loading one file per layer shape (``spconv-test.py:63-73``).
"""
from __future__ import annotations

import math

import torch

from . import _native, backend

__all__ = ["sparse_conv", "sparse_conv_inference", "SparseConv3d", "SparseUNet"]


def sparse_conv(feats: torch.Tensor, weight: torch.Tensor, kmap, arch80: bool = True) -> torch.Tensor:
    """``out[omap[j]] += feats[imap[j]] @ weight[k(j)]`` over the pairs of ``kmap``; differentiable."""
    if feats.size(0) != kmap.n_in:
        raise ValueError(f"feats has {feats.size(0)} rows, the kernel map expects {kmap.n_in}")
    if weight.size(0) != kmap.kpos.numel() - 1:
        raise ValueError("weight and kernel map disagree on the number of offsets")
    return _native.sparse_conv(feats, weight, kmap.kpos, kmap.imap, kmap.omap, kmap.n_out, arch80)


def sparse_conv_inference(feats: torch.Tensor, weight: torch.Tensor, kmap, bias: torch.Tensor | None = None,
                          relu: bool = False, arch80: bool = True) -> torch.Tensor:
    """Forward only, through the output-stationary kernel (``backend.fgms_fwd_os_cuda``): every output row is
    written once — the same bits on every run — with ``bias`` and ReLU applied in the kernel's epilogue (a
    batch-norm layer in inference form is a scaled weight and a bias).  No autograd.  The neighbour table the
    kernel reads is built on first use and kept on ``kmap``.  Tensor-core shapes only (fp16, or fp32 storage
    with tf32 arithmetic; channel counts multiples of 16 up to 256)."""
    if feats.size(0) != kmap.n_in:
        raise ValueError(f"feats has {feats.size(0)} rows, the kernel map expects {kmap.n_in}")
    nbr = getattr(kmap, "_neighbor_table", None)
    if nbr is None:
        nbr = backend.build_neighbor_table(kmap.kpos, kmap.imap, kmap.omap, kmap.n_in, kmap.n_out)
        try:
            kmap._neighbor_table = nbr
        except AttributeError:  # a map type without room for it: rebuilt on every call
            pass
    out = torch.empty((kmap.n_out, weight.size(2)), dtype=feats.dtype, device=feats.device)
    with torch.no_grad():
        backend.fgms_fwd_os_cuda(feats.contiguous(), weight.detach().contiguous(), out, nbr, arch80, bias=bias, relu=relu)
    return out


class SparseConv3d(torch.nn.Module):
    """Sparse 3-D convolution layer with a ``[k_vol, c_in, c_out]`` weight (no bias, like the reference's
    operator); initialised like ``torch.nn.Conv3d`` (kaiming uniform, a = sqrt(5), fan_in = c_in * k_vol)."""

    def __init__(self, c_in: int, c_out: int, k_vol: int = 27, dtype=torch.float16, device="cuda", arch80: bool = True):
        super().__init__()
        self.c_in, self.c_out, self.k_vol, self.arch80 = c_in, c_out, k_vol, arch80
        bound = 1.0 / math.sqrt(c_in * k_vol)
        w = (torch.rand((k_vol, c_in, c_out), device=device, dtype=torch.float32) * 2 - 1) * bound
        self.weight = torch.nn.Parameter(w.to(dtype))

    def forward(self, feats: torch.Tensor, kmap) -> torch.Tensor:
        return sparse_conv(feats, self.weight, kmap, self.arch80)


_LAYER_FORWARD = SparseConv3d.forward
_MODULE = torch.nn.modules.module
_HOOKS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")


def _watched() -> bool:
    """Whether something beyond the layers themselves sees or transforms their calls.  PyTorch answers most of this under private names
    only: a release that lacks one counts as watching.  Several ranks count too, because gradients that leave with their layer are
    exchanged beside the rest of the backward."""
    try:
        return (torch._C._get_tracing_state() is not None or torch.compiler.is_compiling() or torch.autograd.forward_ad._current_level >= 0
                or torch._C._functorch.peek_interpreter_stack() is not None
                or torch._C._autograd._top_saved_tensors_default_hooks(True) is not None
                or torch._C._len_torch_dispatch_stack() > 0 or torch._C._len_torch_function_stack() > 0
                or (torch.distributed.is_available() and torch.distributed.is_initialized())
                or bool(_MODULE._global_forward_hooks or _MODULE._global_forward_pre_hooks
                        or _MODULE._global_backward_hooks or _MODULE._global_backward_pre_hooks))
    except AttributeError:
        return True


def _one_node(layers) -> bool:
    """Whether a stack may run as one autograd node: nothing sees the calls of its layers."""
    if _watched() or SparseConv3d.forward is not _LAYER_FORWARD or SparseConv3d.__call__ is not torch.nn.Module.__call__:
        return False
    for layer in layers:
        d = layer.__dict__
        if type(layer) is not SparseConv3d or "forward" in d or d["arch80"] != layers[0].__dict__["arch80"] or any(d.get(h, True) for h in _HOOKS):
            return False
    return True


class SparseUNet(torch.nn.Module):
    """The encoder-decoder stack of :mod:`fgms_b200.unet` as an ``nn.Module`` over the autograd operator: one
    :class:`SparseConv3d` per layer of the specification, decoder skips added to the transposed convolutions'
    outputs.  ``forward(feats, umaps)`` takes the kernel maps of all resolutions (``unet.build_unet_maps``)."""

    def __init__(self, spec, dtype=torch.float16, device="cuda", arch80: bool = True):
        super().__init__()
        self.spec = list(spec)
        self.layers = torch.nn.ModuleList(
            SparseConv3d(l.c_in, l.c_out, l.k_vol, dtype=dtype, device=device, arch80=arch80) for l in self.spec)

    def load_weights(self, weights):
        with torch.no_grad():
            for layer, w in zip(self.layers, weights):
                layer.weight.copy_(torch.as_tensor(w).to(layer.weight.device, layer.weight.dtype))

    def _forward_as_one(self, feats: torch.Tensor, umaps):
        """The stack as one autograd node (``csrc/torch_binding.cpp``), or None: see :func:`_one_node`."""
        layers = list(self.layers)
        if not layers or len(layers) != len(self.spec) or type(feats) is not torch.Tensor or not _one_node(layers):
            return None
        value, seen, weights, maps, plan = {"input": 0}, {}, [], [], []
        for spec, layer in zip(self.spec, layers):
            w, km = layer._parameters.get("weight"), umaps.of(spec)
            if type(w) is not torch.nn.Parameter or spec.src not in value or (spec.skip is not None and spec.skip not in value):
                return None
            m, _ = seen.setdefault(id(km), (len(seen), km))  # with the map itself: an id is one object's for as long as it lives
            if 3 * m == len(maps):
                maps += km.kpos, km.imap, km.omap
            plan += value[spec.src], -1 if spec.skip is None else value[spec.skip], m, km.n_in, km.n_out
            weights.append(w)
            value[spec.dst] = len(weights)
        if not all(type(t) is torch.Tensor for t in maps):
            return None
        return _native.sparse_stack(feats, weights, maps, plan, layers[0].arch80)

    def forward(self, feats: torch.Tensor, umaps) -> torch.Tensor:
        out = self._forward_as_one(feats, umaps)
        if out is not None:
            return out
        val = {"input": feats}
        for spec, layer in zip(self.spec, self.layers):
            y = layer(val[spec.src], umaps.of(spec))
            if spec.skip is not None:
                y = y + val[spec.skip]
            val[spec.dst] = y
        return val[self.spec[-1].dst]
