"""Layer calls without the module machinery, for networks whose iteration is
bound by host time.

``nn.Module.__call__`` and the layers' own Python cost 4 to 8 us per layer, a
fifth of ResNet-20's forward pass on the host.  ``conv`` and ``batch_norm`` make
the layer's one library call directly when nothing observes or replaces it: a
plain layer without hooks (its own or global ones), whose forward is neither
replaced (on the instance or for the class) nor compiled, called with a tensor
outside of tracing.  Otherwise they call the layer.  (Code that is itself
scripted or compiled calls the layers: the caller's check, once per block.)
``sequence`` does the same for the batch norms of an ``nn.Sequential``.
"""
from __future__ import annotations

import contextlib
import threading

import torch
import torch.nn as nn
from torch.nn.modules import module as _m

_Module, _Conv2d, _BatchNorm2d = nn.Module, nn.Conv2d, nn.BatchNorm2d
_call, _conv_forward, _bn_forward = nn.Module.__call__, nn.Conv2d.forward, nn.BatchNorm2d.forward
_sequence_forward = nn.Sequential.forward
_tracing = torch._C._get_tracing_state


def _plain(layer: nn.Module) -> bool:
    own = layer.__dict__
    return not (layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks or layer._backward_pre_hooks
                or _m._global_forward_hooks or _m._global_forward_pre_hooks or _m._global_backward_hooks
                or _m._global_backward_pre_hooks
                or "forward" in own or "_conv_forward" in own or "_check_input_dim" in own
                or own.get("_compiled_call_impl") is not None or _Module.__call__ is not _call or _tracing() is not None)


class _Gathered(threading.local):
    counters = None   # of the batch-norm layers called so far, where this thread gathers them


_gathered = _Gathered()


@contextlib.contextmanager
def gathered_counters():
    """Within, the ``num_batches_tracked`` counters of the layers that
    ``batch_norm`` calls directly are advanced by one launch at the end instead of
    one per layer (8 us of host time each).  Each call counts once, as it would
    have by itself; until the end the counters are behind by this pass."""
    outer, mine = _gathered.counters, []
    _gathered.counters = mine
    try:
        yield
    finally:
        _gathered.counters = outer
        if len({c.data_ptr() for c in mine}) == len(mine):
            if mine:
                torch._foreach_add_(mine, 1)
        else:   # a layer that ran twice, or two that share a counter: one launch would lose a count
            for c in mine:
                c.add_(1)


def layers_of(module: nn.Module, *names):
    """The module's attributes of these names, without ``__getattr__`` where they are registered layers."""
    registered = module._modules
    try:
        return [registered[n] for n in names]
    except KeyError:
        return [getattr(module, n) for n in names]


def conv(layer: nn.Module, x):
    if type(layer) is _Conv2d and isinstance(x, torch.Tensor) and layer.padding_mode == "zeros" \
            and _Conv2d.forward is _conv_forward and _plain(layer):
        p = layer._parameters
        if "weight" in p and "bias" in p:
            return torch.conv2d(x, p["weight"], p["bias"], layer.stride, layer.padding, layer.dilation, layer.groups)
    return layer(x)


def batch_norm(layer: nn.Module, x):
    if type(layer) is _BatchNorm2d and isinstance(x, torch.Tensor) and layer.training and layer.track_running_stats \
            and layer.momentum is not None and x.dim() == 4 and x.numel() > x.size(1) \
            and _BatchNorm2d.forward is _bn_forward and _plain(layer):
        p, b = layer._parameters, layer._buffers
        if "weight" in p and "bias" in p and "num_batches_tracked" in b and b.get("running_mean") is not None \
                and b.get("running_var") is not None:
            counter = b["num_batches_tracked"]
            if counter is not None:
                if _gathered.counters is None:
                    counter.add_(1)
                else:
                    _gathered.counters.append(counter)
            return torch.batch_norm(x, p["weight"], p["bias"], b["running_mean"], b["running_var"], True, layer.momentum,
                                    layer.eps, torch.backends.cudnn.enabled)
    return layer(x)


def sequence(layers: nn.Module, x):
    if type(layers) is nn.Sequential and isinstance(x, torch.Tensor) and nn.Sequential.forward is _sequence_forward \
            and _plain(layers):
        for layer in layers._modules.values():
            x = batch_norm(layer, x) if type(layer) is _BatchNorm2d else layer(x)
        return x
    return layers(x)
