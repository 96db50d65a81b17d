"""Typed tensor transfer on one device (or from pinned host memory to the device) over the native kernels.

Same contract as the reference's ``copy_tensor`` and ``TensorTransfer``
(vllm_rlt/worker/tensors.py:35-87, :282-365): equal-sized contiguous tensors for the flat copy, batches of
disjoint 1-D/2-D copies of one (source type, target type) pair for the segmented one, the five transfer
dtypes, and the same ``ValueError`` conditions, including the refusal of copies between two different CUDA
devices (those go through the handoff connector). There is no CPU or PyTorch fallback here: targets must be
CUDA tensors and host sources must be pinned.
"""

from __future__ import annotations

import torch

from .. import _lib

_DTYPES = {torch.int32: 0, torch.int64: 1, torch.float16: 2, torch.bfloat16: 3, torch.float32: 4}


def copy_tensor(source: torch.Tensor, target: torch.Tensor, *, secondary: torch.Tensor | None = None) -> torch.Tensor:
    """Copy contiguous values to their final storage, optionally writing a second typed output."""
    _lib.check(_lib.load_host().tensor_copy(source, target, secondary), "rlt_tensor_copy")
    return target


class TensorTransfer:
    """One typed batch of disjoint 1-D/2-D copies with borrowed tensor references.

    ``append`` records a copy, ``submit`` launches the whole batch as one kernel, ``reset`` forgets it.
    The descriptors of a batch of up to 448 copies between tensors of one type are parameters of the launch; others are
    written into a pinned table that the kernel reads through its device mapping. Either way a submission needs no
    separate host-to-device copy. The table and the tensors of a submitted batch must stay untouched until the work
    queued behind ``submit`` has completed.
    """

    def __init__(self, capacity: int, dtype: torch.dtype, device, *, target_dtype: torch.dtype | None = None):
        self.dtype, self.target_dtype = dtype, target_dtype or dtype
        if self.dtype not in _DTYPES or self.target_dtype not in _DTYPES:
            raise ValueError("unsupported transfer dtype")
        self.device = torch.device(device)
        if self.device.type != "cuda":
            raise ValueError("transfer destination must be a CUDA device")
        self._index = -1 if self.device.index is None else self.device.index  # no tensor is on a device without index
        self.capacity = capacity
        self.table = torch.zeros((capacity, 8), dtype=torch.int64, pin_memory=True)
        host = _lib.load_host()
        self._rows = host.transfer_new()
        self._append, self._submit, self._reset = host.transfer_append, host.transfer_submit, host.transfer_reset
        self._types = _DTYPES[self.dtype], _DTYPES[self.target_dtype]
        self.reset()

    def reset(self) -> None:
        self.copies: list[tuple[torch.Tensor, torch.Tensor]] = []
        self._reset(self._rows)

    def append(self, source: torch.Tensor, target: torch.Tensor) -> None:
        if self._append(self._rows, self.capacity, *self._types, self._index, source, target):
            self.copies.append((source, target))

    def submit(self) -> None:
        if self.copies:
            _lib.check(self._submit(self._rows, *self._types, self._index, self.table), "rlt_tensor_transfer")

    @property
    def max_rows(self) -> int:
        return _lib.load_host().transfer_extent(self._rows)[0]

    @property
    def max_cols(self) -> int:
        return _lib.load_host().transfer_extent(self._rows)[1]
