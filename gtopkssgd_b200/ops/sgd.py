"""K3 wrapper: fused sparse scatter + averaging + weight decay + momentum SGD.

``sgd_dense`` applies the part of the update that does not depend on the
sparse exchange (weight decay, momentum decay, and the dense gradient in dense
mode); ``sgd_sparse`` applies the k global pairs on top.  Together they equal
the reference's scatter + ``/P`` + per-parameter SGD loop
(allreducer.py:458-475, distributed_optimizer.py:105-143).  CPU tensors go
through the PyTorch oracle.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Optional

import torch

from . import lib as _lib
from . import oracle
from .select import _ptr, _raw_stream, current_stream_handle, pairs_to_tensors


@dataclass
class SgdHyper:
    lr: float
    momentum: float = 0.0
    dampening: float = 0.0
    weight_decay: float = 0.0
    nesterov: bool = False


def sgd_dense(p: torch.Tensor, buf: Optional[torch.Tensor], h: SgdHyper, first_step: bool,
              g: Optional[torch.Tensor] = None, scale: float = 1.0, coef: Optional[torch.Tensor] = None,
              lr_dev: Optional[torch.Tensor] = None) -> None:
    """Dense part of the step over a flat parameter buffer.  With ``g`` given
    (dense mode) the gradient is ``coef * scale * g``."""
    d = p.numel()
    if p.device.type != "cuda":
        if g is None and h.momentum == 0 and h.weight_decay == 0:
            return
        c = scale * (float(coef) if coef is not None else 1.0)
        grad = g * c if g is not None else torch.zeros_like(p)
        oracle.sgd_step(p, buf, grad, h.lr, h.momentum, h.dampening, h.weight_decay, h.nesterov, first_step)
        return
    code = _lib.calls().gtk_k3_dense(p.data_ptr(), _ptr(buf), _ptr(g), _ptr(coef), scale, d, h.lr, _ptr(lr_dev),
                                     h.momentum, h.dampening, h.weight_decay, int(h.nesterov), int(first_step),
                                     current_stream_handle(p.device))
    if code:
        _lib.check(code, "gtk_k3_dense")


def sgd_sparse(p: torch.Tensor, buf: Optional[torch.Tensor], pairs: torch.Tensor, counts: torch.Tensor,
               nseg: int, seg_stride: int, h: SgdHyper, first_step: bool, scale: float,
               coef: Optional[torch.Tensor] = None, use_atomics: bool = False,
               bad_index_count: Optional[torch.Tensor] = None, lr_dev: Optional[torch.Tensor] = None,
               parity_word: Optional[torch.Tensor] = None, parity_stride: int = 0, max_count: int = 0) -> None:
    """Sparse part of the step: for every pair (j, v) of every segment add
    ``coef * scale * v`` as gradient of element j.  ``counts`` is a device
    tensor with the live length of each segment.  ``lr_dev`` (a device scalar)
    overrides ``h.lr``; ``parity_word`` selects the half of a two-parity buffer
    on the device: base = pairs + ((word - 1) & 1) * parity_stride.
    ``max_count``: how long a segment's list is expected to be at most, where
    the caller knows it to be shorter than ``seg_stride`` (0: not known); it
    decides how much is launched, not what is applied."""
    d = p.numel()
    if not p.is_cuda:
        if parity_word is not None:
            pairs = pairs[((int(parity_word) - 1) & 1) * parity_stride:]
        c = scale * (float(coef) if coef is not None else 1.0)
        f = 1.0 if first_step else 1.0 - h.dampening
        for s in range(nseg):
            n = int(counts[s])
            idx, val = pairs_to_tensors(pairs[s * seg_stride:(s + 1) * seg_stride], n)
            sv = val * c
            step = sv
            if h.momentum != 0 and buf is not None:
                sb = f * sv
                buf.index_add_(0, idx, sb)
                step = sv + h.momentum * sb if h.nesterov else sb
            p.index_add_(0, idx, step, alpha=-h.lr)
        return
    index = p.get_device()
    if bad_index_count is None:
        bad = _scratch_addresses.get(index) or _scratch_address(index)
    else:
        bad = bad_index_count.data_ptr()
    # how many pairs may be read, valid or not (0: not known): an expanded view, or another whose elements do not lie side
    # by side, has more bytes than there is memory behind it
    readable = pairs.nbytes >> 3 if pairs.is_contiguous() else 0
    code = _lib.calls().gtk_k3_sparse(p.data_ptr(), None if buf is None else buf.data_ptr(), pairs.data_ptr(),
                                      counts.data_ptr(), nseg, seg_stride, None if coef is None else coef.data_ptr(),
                                      scale, d, h.lr, None if lr_dev is None else lr_dev.data_ptr(), h.momentum,
                                      h.dampening, h.weight_decay, 1 if h.nesterov else 0, 1 if first_step else 0,
                                      1 if use_atomics else 0, bad,
                                      None if parity_word is None else parity_word.data_ptr(), parity_stride,
                                      readable, max_count, _raw_stream(index))
    if code:
        _lib.check(code, "gtk_k3_sparse")


def scatter_dense(g: torch.Tensor, pairs: torch.Tensor, counts: torch.Tensor, nseg: int, seg_stride: int,
                  scale: float, use_atomics: bool = False, parity_word: Optional[torch.Tensor] = None,
                  parity_stride: int = 0) -> None:
    """g <- 0, then g[j] (+)= scale * v for every pair: the dense averaged
    gradient, for callers that want to inspect ``p.grad``."""
    if g.device.type != "cuda":
        if parity_word is not None:
            pairs = pairs[((int(parity_word) - 1) & 1) * parity_stride:]
        g.zero_()
        for s in range(nseg):
            n = int(counts[s])
            idx, val = pairs_to_tensors(pairs[s * seg_stride:(s + 1) * seg_stride], n)
            g.index_add_(0, idx, val * scale)
        return
    code = _lib.calls().gtk_k3_scatter_dense(g.data_ptr(), pairs.data_ptr(), counts.data_ptr(), nseg, seg_stride, scale,
                                             g.numel(), int(use_atomics), _ptr(parity_word), parity_stride,
                                             current_stream_handle(g.device))
    if code:
        _lib.check(code, "gtk_k3_scatter_dense")


_scratch = {}
_scratch_addresses = {}


def _scratch_word(device: torch.device) -> torch.Tensor:
    word = _scratch.get(device)
    if word is None:
        word = _scratch[device] = torch.zeros(1, dtype=torch.int32, device=device)
    return word


def _scratch_address(index: int) -> int:
    at = _scratch_addresses.get(index)
    if at is None:
        at = _scratch_addresses[index] = _scratch_word(torch.device("cuda", index)).data_ptr()
    return at


def momentum_correct(v: torch.Tensor, g: torch.Tensor, momentum: float) -> None:
    """v = momentum * v + g; g = v, in place over flat buffers (one launch).
    The reference applies this per parameter in its gradient hook when
    ``momentum_correction`` is set (distributed_optimizer.py:81-88)."""
    if g.device.type != "cuda":
        v.mul_(momentum).add_(g)
        g.copy_(v)
        return
    code = _lib.calls().gtk_k3_momentum_correct(v.data_ptr(), g.data_ptr(), momentum, g.numel(),
                                                current_stream_handle(g.device))
    if code:
        _lib.check(code, "gtk_k3_momentum_correct")
