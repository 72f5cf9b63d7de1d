"""Top-1 accuracy of a batch in one launch (K5)."""
from __future__ import annotations

import torch

from . import lib as _lib
from .select import current_stream_handle

MAX_ELEMENTS = 1 << 18  # one CTA reads the logits; larger batches take the library's way


def takes(output: torch.Tensor, target: torch.Tensor) -> bool:
    return (output.is_cuda and output.dim() == 2 and output.dtype == torch.float32 and output.is_contiguous()
            and output.get_device() == torch.cuda.current_device()  # a launch goes to the current device
            and 0 < output.numel() <= MAX_ELEMENTS and target.dtype == torch.int64 and target.is_contiguous()
            and target.numel() == output.size(0) and target.device == output.device)


def top1_percent(output: torch.Tensor, target: torch.Tensor) -> torch.Tensor:
    """Per cent of rows whose largest logit is the target's, as a tensor of one element."""
    out = torch.empty(1, dtype=torch.float32, device=output.device)
    rows = output.size(0)
    code = _lib.calls().gtk_k5_top1(output.data_ptr(), target.data_ptr(), rows, output.size(1), 100.0 / rows, out.data_ptr(),
                                    current_stream_handle(output.device))
    if code:
        _lib.check(code, "gtk_k5_top1")
    return out
