"""Layer calls without the module machinery, for networks whose iteration is
bound by host time.

``nn.Module.__call__`` and the layers' own Python cost 4 to 8 us per layer, a
fifth of ResNet-20's forward pass on the host.  ``conv`` and ``batch_norm`` make
the layer's one library call directly when nothing observes or replaces it: a
plain layer without hooks (its own or global ones), called with a tensor, outside
of scripting.  Otherwise they call the layer.
"""
from __future__ import annotations

import torch
import torch.nn as nn
from torch.nn.modules import module as _m


def _plain(layer: nn.Module) -> bool:
    return not (layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks or layer._backward_pre_hooks
                or _m._global_forward_hooks or _m._global_forward_pre_hooks or _m._global_backward_hooks
                or _m._global_backward_pre_hooks)


def conv(layer: nn.Module, x):
    if type(layer) is nn.Conv2d and isinstance(x, torch.Tensor) and layer.padding_mode == "zeros" and _plain(layer):
        p = layer._parameters
        if "weight" in p:
            return torch.conv2d(x, p["weight"], p["bias"], layer.stride, layer.padding, layer.dilation, layer.groups)
    return layer(x)


def batch_norm(layer: nn.Module, x):
    if type(layer) is nn.BatchNorm2d and isinstance(x, torch.Tensor) and layer.training and layer.track_running_stats \
            and layer.momentum is not None and x.dim() == 4 and x.numel() > x.size(1) and _plain(layer):
        p, b = layer._parameters, layer._buffers
        if "weight" in p and b.get("running_mean") is not None:
            counter = b["num_batches_tracked"]
            if counter is not None:
                counter.add_(1)
            return torch.batch_norm(x, p["weight"], p["bias"], b["running_mean"], b["running_var"], True, layer.momentum,
                                    layer.eps, torch.backends.cudnn.enabled)
    return layer(x)
