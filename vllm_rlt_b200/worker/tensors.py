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


def _transfer_type():
    class TensorTransfer(_lib.load_host().Copies):
        """One typed batch of disjoint 1-D/2-D copies with borrowed tensor references.

        ``append(source, target)`` records a copy in ``copies``, ``submit`` launches the whole batch as one kernel, ``reset``
        forgets it (``append`` and ``reset`` are the compiled base's, which holds the descriptors).
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
            self.table = torch.zeros((capacity, 8), dtype=torch.int64, pin_memory=True)
            # no tensor is on a device without index
            self.setup(capacity, _DTYPES[self.dtype], _DTYPES[self.target_dtype], -1 if self.device.index is None else self.device.index)

        def submit(self) -> None:
            _lib.check(self.launch(self.table), "rlt_tensor_transfer")

    return TensorTransfer


__getattr__ = _lib.on_demand(globals(), TensorTransfer=_transfer_type)
