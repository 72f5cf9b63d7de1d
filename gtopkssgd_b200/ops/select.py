"""K1 wrapper: fused residual add + top-k select + residual write-back.

``TopkSelector`` owns the device buffers of one merged gradient group (the
candidate list, the selected pairs, the persistent threshold state and the
control block) and enqueues the two K1 launches on the current stream.  On CPU
tensors it runs the PyTorch oracle instead, with the same outputs.
"""
from __future__ import annotations

import math
from typing import Optional, Sequence, Tuple

import torch

from . import lib as _lib
from . import oracle


_FLOAT = torch.float32


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


# the handle of the current stream of a device index, without building a Stream object (0.1 us against 3 us)
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def current_stream_handle(device: torch.device) -> int:
    index = device.index
    return _raw_stream(torch.cuda.current_device() if index is None else index)


class TopkSelector:
    """Per-group selection state.

    Pairs are stored as an int32 tensor of shape [n, 2]: column 0 is the index,
    column 1 holds the fp32 value bits.
    """

    def __init__(self, numel: int, max_k: int, device: torch.device, target_ratio: float = 3.0,
                 cap_factor: int = 32, limit_ms: float = 2000.0):
        if numel >= 2 ** 31:
            raise ValueError("a merged group must have fewer than 2^31 elements")
        self.numel = int(numel)
        self.max_k = int(min(max_k, numel))
        self.device = torch.device(device)
        self.target_ratio = float(target_ratio)
        self.limit_ns = int(limit_ms * 1e6)
        self.cap = int(max(self.max_k, min(self.numel, max(cap_factor * self.max_k, 4096))))
        self.is_cuda = self.device.type == "cuda"
        self.sel = torch.zeros((self.max_k, 2), dtype=torch.int32, device=self.device)
        self.state = torch.zeros(16, dtype=torch.int32, device=self.device)
        self._n_sel = self.state[1:2]   # (a view costs over 1 us to make)
        self.reset_threshold()
        if self.is_cuda:
            L = _lib.lib()
            assert L.gtk_k1state_bytes() == 64
            self.cand = torch.empty((self.cap, 2), dtype=torch.int32, device=self.device)
            # two control blocks: call i uses block i & 1 and clears the other one for call i + 1
            self.ctrl_words = int(L.gtk_ctrl_bytes()) // 4
            self.ctrl = torch.zeros(2 * self.ctrl_words, dtype=torch.int32, device=self.device)
            self._stream_index = self.sel.device.index
            self._select = _lib.calls().gtk_k1_select
            self._select_segments = _lib.calls().gtk_k1_select_segments
            self._compress = _lib.calls().gtk_k1_compress
            self._buffers = (self.cand.data_ptr(), self.cap, self.sel.data_ptr(), self.state.data_ptr(),
                             self.ctrl.data_ptr(), self.target_ratio, self.limit_ns)
        self.last_k = 0

    # -- state ---------------------------------------------------------------
    def reset_threshold(self) -> None:
        """Forget the predicted threshold: the next call takes the exact path."""
        self.state.view(torch.float32)[0] = math.inf

    @property
    def n_sel_tensor(self) -> torch.Tensor:
        """Device word holding the number of selected pairs of the last call."""
        return self._n_sel

    def stats(self) -> dict:
        """Host copy of the selection statistics (synchronises)."""
        s = self.state.cpu()
        f = s.view(torch.float32)
        return {"tau": float(f[0]), "n_sel": int(s[1]), "n_cand": int(s[2]), "fallback": int(s[3]),
                "n_fallbacks": int(s[4]), "n_calls": int(s[5]), "kth_mag": float(f[6])}

    def status(self) -> Tuple[int, int]:
        """(status, code location) of the last failure in either control block,
        (0, 0) if none.  Synchronises."""
        if not self.is_cuda:
            return (0, 0)
        for b in (0, 1):
            c = self.ctrl[b * self.ctrl_words:b * self.ctrl_words + 8].cpu()
            if int(c[_lib.CTRL_STATUS]):
                return int(c[_lib.CTRL_STATUS]), int(c[_lib.CTRL_WHERE])
        return (0, 0)

    def trace(self) -> dict:
        """Device-side phase stamps of the last select, in nanoseconds since its
        start: slot 1 = CTA 0 finished its share of the stream pass, 2 = the pick
        began, 3 = k-th magnitude or its bin known (where all CTAs share the candidates), 4 = winners
        compacted (2 to 4 only when the prediction held).  Synchronises."""
        if not self.is_cuda:
            return {}
        calls = int(self.state[5].item())
        b = (calls - 1) & 1
        return _lib.read_trace(self.ctrl[b * self.ctrl_words:(b + 1) * self.ctrl_words])

    def reset(self) -> None:
        """Back to the initial state (after a reported failure)."""
        if self.is_cuda:
            self.ctrl.zero_()
        self.state.zero_()
        self.reset_threshold()

    # -- the op ----------------------------------------------------------------
    def select(self, g: torch.Tensor, r: torch.Tensor, k: int, g_scale: Optional[torch.Tensor] = None) -> None:
        """acc = g*scale + r; self.sel[:k] <- the k largest-magnitude (idx, acc)
        pairs; r <- acc off the selection, 0 on it.  g is not modified."""
        numel = self.numel
        assert g.numel() == numel and r.numel() == numel
        assert g.dtype is _FLOAT and r.dtype is _FLOAT
        k = int(k if k < self.max_k else self.max_k)
        self.last_k = k
        if not self.is_cuda:
            scale = float(g_scale) if g_scale is not None else 1.0
            idx, val = oracle.compress(g.view(-1), r.view(-1), k, scale)
            self.sel[:k, 0] = idx.to(torch.int32)
            self.sel[:k, 1] = val.view(torch.int32)
            self.state[1] = k
            return
        assert g.is_contiguous() and r.is_contiguous()
        code = self._select(g.data_ptr(), r.data_ptr(), None if g_scale is None else g_scale.data_ptr(), numel, k,
                            *self._buffers, _raw_stream(self._stream_index))
        if code:
            _lib.check(code, "gtk_k1_select")

    def select_segments(self, addresses: Sequence[int], segments: torch.Tensor, r: torch.Tensor, k: int) -> None:
        """``select`` (CUDA only) with the gradient in one tensor per parameter:
        ``addresses`` are their device addresses (0: no gradient), ``segments`` an
        int32 device tensor with the n + 1 start positions in float4 and the n
        lengths in elements (see ``segment_table``)."""
        assert r.numel() == self.numel and r.dtype is _FLOAT and r.is_contiguous()
        assert segments.numel() == 2 * len(addresses) + 1 and segments.dtype is torch.int32 and segments.is_contiguous()
        k = int(min(k, self.max_k))
        self.last_k = k
        code = self._select_segments(addresses, segments.data_ptr(), r.data_ptr(), self.numel, k, *self._buffers,
                                     _raw_stream(self._stream_index))
        if code:
            _lib.check(code, "gtk_k1_select_segments")

    def compress(self, g: torch.Tensor, r: torch.Tensor, k: int) -> Tuple[torch.Tensor, torch.Tensor]:
        """``select`` that also leaves g sparsified (acc on the selection, 0 off
        it) and returns the selection as (int64 indices, fp32 values).  Nothing
        synchronises: the number of selected entries is min(k, numel)."""
        assert g.numel() == self.numel and r.numel() == self.numel
        assert g.dtype is _FLOAT and r.dtype is _FLOAT
        assert g.is_contiguous() and r.is_contiguous()
        k = int(min(k, self.max_k))
        self.last_k = k
        idx = torch.empty(k, dtype=torch.int64, device=g.device)
        val = torch.empty(k, dtype=torch.float32, device=g.device)
        code = self._compress(g.data_ptr(), r.data_ptr(), self.numel, k, *self._buffers, idx.data_ptr(),
                              val.data_ptr(), _raw_stream(self._stream_index))
        if code:
            _lib.check(code, "gtk_k1_compress")
        return idx, val

    def pairs(self) -> Tuple[torch.Tensor, torch.Tensor]:
        """(int64 indices, fp32 values) of the last selection (synchronises)."""
        n = int(self.state[1].item())
        p = self.sel[:n]
        return p[:, 0].to(torch.int64), p[:, 1].contiguous().view(torch.float32)


MAX_SEGMENTS = 1024  # gradient tensors that one select can take


def segment_table(offsets: Sequence[int], sizes: Sequence[int], numel: int, device: torch.device) -> torch.Tensor:
    """The table that ``TopkSelector.select_segments`` reads, for parameters at
    ``offsets`` (multiples of 4, without gaps of a whole float4) of a flat
    vector of ``numel`` elements."""
    assert all(o % 4 == 0 for o in offsets)
    starts = [o // 4 for o in offsets] + [(numel + 3) // 4]
    return torch.tensor(starts + list(sizes), dtype=torch.int32, device=device)


def pairs_to_tensors(pairs: torch.Tensor, n: int) -> Tuple[torch.Tensor, torch.Tensor]:
    p = pairs[:n]
    return p[:, 0].to(torch.int64), p[:, 1].contiguous().view(torch.float32)


def tensors_to_pairs(idx: torch.Tensor, val: torch.Tensor, out: torch.Tensor) -> int:
    n = idx.numel()
    out[:n, 0] = idx.to(torch.int32)
    out[:n, 1] = val.to(torch.float32).view(torch.int32)
    return n
