"""Python face of the KV-handoff kernels: argument checking and the C-ABI calls.

These wrappers play the role that ``vllm_rlt/kernels/activation.py`` plays for
the reference's one native op: validate on the host, then launch on the
caller's current CUDA stream without synchronising. There is no fallback: if
the native library is not built, or no CUDA device is present, the calls raise.

Reference behaviour that is kept: bad ranges and tables raise ``ValueError``
with the messages of ``kv_segments`` (vllm_rlt/pd/transport.py:29-47).
"""

from __future__ import annotations

import contextlib
import ctypes as C
import threading
from dataclasses import dataclass, field
from typing import Sequence

import numpy as np
import torch

from .. import _lib
from .._lib import MODE_ALL_PLANES, MODE_DEDUP, MODE_EXIT_ONLY  # noqa: F401  (re-exported)


def _stream_ptr(stream) -> int:
    if stream is None:
        return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device())
    if isinstance(stream, int):
        return stream
    return stream.cuda_stream


def _on_stream(address: int):
    """Context in which the stream at ``address`` is the current device's current one. (``ExternalStream`` takes no address of 0: it
    makes a new stream then.)"""
    if address == _stream_ptr(None):
        return contextlib.nullcontext()
    return torch.cuda.stream(torch.cuda.default_stream() if address in (0, 1) else torch.cuda.ExternalStream(address))


def _raw_stream(stream):
    """``stream`` as the compiled host side takes it: an address, or None for the current stream."""
    return stream if stream is None or isinstance(stream, int) else stream.cuda_stream


# --------------------------------------------------------------------------- pools


@dataclass(frozen=True)
class Region:
    """One K/V tensor pair as raw pointers and byte strides (``_kv_region``, vllm_rlt/pd/transport.py:18-26)."""

    key_ptr: int
    value_ptr: int
    block_bytes: int
    layer_bytes: int
    token_bytes: int

    @classmethod
    def of(cls, key: torch.Tensor, value: torch.Tensor) -> "Region":
        if key.shape != value.shape or key.dtype != value.dtype or key.device != value.device:
            raise ValueError("key and value tensors must agree in shape, dtype and device")
        if key.dim() < 4 or not key.is_contiguous() or not value.is_contiguous():
            raise ValueError("pool tensors must be contiguous [blocks, layers, block_size, ...]")
        e = key.element_size()
        return cls(key.data_ptr(), value.data_ptr(), key.stride(0) * e, key.stride(1) * e, key.stride(2) * e)

    def rebased(self, key_ptr: int, value_ptr: int) -> "Region":
        return Region(key_ptr, value_ptr, self.block_bytes, self.layer_bytes, self.token_bytes)

    def as_struct(self) -> _lib.RltRegion:
        return _lib.RltRegion(self.key_ptr, self.value_ptr, self.block_bytes, self.layer_bytes, self.token_bytes)


_NO_REGION = _lib.RltRegion(None, None, 0, 0, 0)


@dataclass(frozen=True)
class PoolView:
    """Geometry and addresses of one paged KV pool, local or mapped from a peer GPU.

    ``scales`` is set only when scale tensors travel: a dynamic-scale FP8 pool.
    A fixed-scale FP8 pool keeps its (constant) scale tensors out of the handoff,
    as the reference does (vllm_rlt/pd/transport.py:132-137).
    """

    codes: Region
    scales: Region | None
    num_blocks: int
    block_size: int
    num_layers: int
    num_planes: int
    device: int
    keepalive: tuple = field(default=(), compare=False, repr=False)

    @classmethod
    def from_tensors(cls, key, value, num_planes, key_scale=None, value_scale=None) -> "PoolView":
        if not key.is_cuda:
            raise ValueError("KV pools must live on a CUDA device: the handoff has no CPU path")
        codes = Region.of(key, value)
        scales = None
        keep = (key, value)
        if key_scale is not None:
            if key_scale.shape != key.shape[:-1] or key_scale.dtype != torch.float32:
                raise ValueError("scale tensors must be float32 [blocks, layers, block_size, kv_heads]")
            scales = Region.of(key_scale, value_scale)
            keep += (key_scale, value_scale)
        return cls(codes, scales, key.shape[0], key.shape[2], key.shape[1], int(num_planes), key.device.index, keep)

    @classmethod
    def from_cache(cls, cache) -> "PoolView":
        """From a ``KVCacheManager``-shaped object (vllm_rlt/core/kv_cache_manager.py:261-271)."""
        dynamic = cache.key_scale is not None and cache.fp8_scale is None
        return cls.from_tensors(
            cache.key_cache,
            cache.value_cache,
            cache.storage_depths,
            cache.key_scale if dynamic else None,
            cache.value_scale if dynamic else None,
        )

    def as_struct(self) -> _lib.RltPool:
        return _lib.RltPool(
            self.codes.as_struct(),
            self.scales.as_struct() if self.scales is not None else _NO_REGION,
            self.num_blocks,
            self.block_size,
            self.num_layers,
            self.num_planes,
        )

    def _address(self) -> int:
        """Address of a struct of this view that lives as long as the view: a launch needs no new one."""
        hit = self.__dict__.get("_struct")
        if hit is None:
            struct = self.as_struct()
            # one struct, also where two threads get here at once: an address that is in use stays good
            hit = self.__dict__.setdefault("_struct", (C.addressof(struct), struct))
        return hit[0]

    @property
    def row_bytes(self) -> int:
        return self.codes.token_bytes + (self.scales.token_bytes if self.scales is not None else 0)

    def payload_bytes(self, tokens: int, planes: int, layers: int | None = None) -> int:
        """Algorithmic payload of ``tokens`` tokens over ``planes`` planes."""
        return 2 * (self.num_layers if layers is None else layers) * self.row_bytes * tokens * planes


# --------------------------------------------------------------------------- batches


class _Staging:
    """One pinned host buffer; reusable once the copy that read it has completed."""

    def __init__(self, pool: "_PinnedPool", capacity: int):
        self.pool = pool
        self.buffer = torch.empty(capacity, dtype=torch.uint8, pin_memory=True)
        self.event = None

    def free(self) -> bool:
        return self.event is None or self.event.query()

    def release(self) -> None:
        self.event = torch.cuda.Event()
        self.event.record()
        self.pool.give(self)


class _PinnedPool:
    """Pinned staging buffers are costly to allocate (a driver call each), so up to ``KEPT`` of them are kept and reused. One that
    has been acquired is out of the pool until it is released: another thread cannot get it meanwhile."""

    KEPT = 64

    def __init__(self):
        self.buffers: list[_Staging] = []
        self._lock = threading.Lock()

    def acquire(self, size: int) -> _Staging:
        with self._lock:
            for i, b in enumerate(self.buffers):
                if b.buffer.numel() >= size and b.free():
                    return self.buffers.pop(i)
        return _Staging(self, 1 << max(16, (size - 1).bit_length()))

    def give(self, b: _Staging) -> None:
        with self._lock:
            if len(self.buffers) < self.KEPT:
                self.buffers.append(b)


_PINNED = _PinnedPool()


class _Sent:
    """Device memory of a batch and the stream it was filled on, which is also the one the allocator takes it back in the order of.

    A use on another stream comes behind the fill alone (``before``), not behind what else that stream has been given since, and the
    memory goes back behind that use (``after``). ``capture``: the graph capture that the fill is part of, 0 for none."""

    def __init__(self, tensor, stream: int, capture: int = 0):
        self.tensor, self.stream, self.capture = tensor, stream, capture
        self._event = _lib.load_host().event
        self._filled = self._event(False, tensor.device.index, stream)
        self._used = {}  # (device, stream) of the launches elsewhere: an event behind the last of them

    def _elsewhere(self, stream: int):
        """The launching device, which is the current one, and the stream, unless they are where the memory was filled."""
        use = torch.cuda.current_device(), stream
        return None if use == (self.tensor.device.index, self.stream) else use

    def before(self, stream: int, capture: int) -> int:
        if capture != self.capture:
            self._filled.synchronize()  # a graph cannot wait for what lies before it: its replays find the memory filled
        else:
            use = self._elsewhere(stream)
            if use is not None:
                self._filled.order(*use)
        return self.tensor.data_ptr()

    def after(self, stream: int, capture: int) -> None:
        use = self._elsewhere(stream)
        if use is not None and not capture:  # (a batch outlives the graphs that use it)
            self._used[use] = self._event(False, *use)

    def __del__(self):
        try:
            capturing = self._used and _lib.load_host().capture(self.stream)
            for event in self._used.values():
                if capturing:  # the stream's next work is a graph's, which cannot wait for this
                    event.synchronize()
                else:
                    event.order(self.tensor.device.index, self.stream)
        except Exception:  # the caller's stream is gone, and with it whatever was queued there
            pass


class HandoffBatch:
    """Per-request tables and ranges of a batch, checked on the host and kept there as the records the kernels read.

    ``src_tables[r]`` / ``dst_tables[r]`` are the per-plane block tables of request
    ``r`` (``plane_block_tables``); ``ranges[r]`` is its token range; ``exit_planes[r]``
    (optional) holds one zero-based exit plane per token position of the request.
    Validation mirrors ``kv_segments``: same conditions, same messages.

    Everything is copied out of the arguments. A batch of up to about a thousand tokens travels as kernel parameters of
    the launches that use it; the records of a larger one are sent to the device here, on ``stream``, in one copy. The
    padded arrays that an ``RltBatch`` points at are made and sent when something asks for them (``as_struct``).

    Any stream and any thread may use a batch. A CUDA graph may use one that was built before it or within its capture; such
    a batch has to be kept, like the pools, for as long as the graph is replayed.
    """

    def __init__(
        self,
        src_tables: Sequence[Sequence[Sequence[int]]] | None,
        dst_tables: Sequence[Sequence[Sequence[int]]] | None,
        ranges: Sequence[tuple[int, int]],
        *,
        block_size: int,
        exit_planes: Sequence[Sequence[int]] | None = None,
        src_blocks: int | None = None,
        dst_blocks: int | None = None,
        device=None,
        stream=None,
    ):
        host = _lib.load_host()
        (self._plan, self.num_requests, self.total_tokens, self.table_width, self.src_planes, self.dst_planes, self.exit_count,
         self.ranges, self.metadata_bytes) = host.plan(src_tables, dst_tables, ranges, exit_planes, block_size, src_blocks,
                                                       dst_blocks, _lib.MAX_REQUESTS)
        self.block_size = block_size
        self.has_exit = exit_planes is not None
        self._planned_exits = self.exit_count
        self._device = device
        self._arrays = {}     # of the RltBatch form, by graph capture (0: none): (device tensor, address of each array, _Sent)
        self._staged = {}     # what has been sent to the device, by the image's planes (0: the records) and graph capture (0: none)
        self._sending = threading.Lock()
        if not host.plan_fits(self._plan, 0):
            self._send(0, self.metadata_bytes, stream)

    def _where(self):
        return torch.device("cuda", torch.cuda.current_device()) if self._device is None else torch.device(self._device)

    def _send(self, planes: int, nbytes: int, stream) -> _Sent:
        """The records (``planes`` 0), or the wire plan of ``planes`` planes, on the device: sent once, and once more by each graph that
        cannot count on that."""
        with self._sending:
            sent = self._staged.get((planes, 0))
            if sent is None:
                with torch.cuda.device(self._where()):
                    at = _stream_ptr(stream)
                    capture = _lib.load_host().capture(at)
                    sent = self._staged.get((planes, capture))
                    if sent is None:
                        with _on_stream(at):  # memory of the stream that fills it
                            tensor = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
                        _lib.check(_lib.load_host().plan_upload(self._plan, planes, tensor.data_ptr(), at), "rlt_stage_upload")
                        sent = self._staged[planes, capture] = _Sent(tensor, at, capture)
        return sent

    def _move(self, direction, src, dst, *, mode, layer_begin=0, layer_end=0, wire_planes=0, plane_begin=0, plane_end=0,
              mask=0, status=None, grid_limit=0, variant=0, workspace=None, packed=0, packed_bytes=0, stream=None) -> int:
        """One launch from this batch's records; ``_lib.MOVE_UNSUITED`` (nothing launched) where they do not serve."""
        if self._plan is None or self.exit_count != self._planned_exits or variant or grid_limit:
            return _lib.MOVE_UNSUITED
        host = _lib.load_host()
        records = wire = wire_bytes = planes = 0
        if direction != _lib.MOVE_DIRECT and mode == MODE_DEDUP:
            planes = (src if direction == _lib.MOVE_PACK else dst).num_planes
            wire_bytes = host.plan_wire(self._plan, planes)
        used, on, capture = (), 0, 0
        if self._staged or (wire_bytes and not host.plan_fits(self._plan, wire_bytes)):
            on = _stream_ptr(stream)
            capture = host.capture(on)
            used = (self._send(0, self.metadata_bytes, stream),)
            records = used[0].before(on, capture)
            if wire_bytes:
                used += (self._send(planes, wire_bytes, stream),)
                wire = used[1].before(on, capture)
        code = host.move(direction, src and src._address(), dst and dst._address(), self._plan, records, wire, mode, layer_begin,
                         layer_end, wire_planes, plane_begin, plane_end, mask, status, grid_limit, variant, workspace, packed,
                         packed_bytes, _raw_stream(stream))
        for sent in used:
            sent.after(on, capture)
        return code

    def _send_arrays(self, capture: int = 0):
        """The padded arrays of the RltBatch form, in one device buffer: one pinned staging buffer, one copy on the current stream."""
        host = _lib.load_host()
        size, offsets = host.plan_layout(self._plan)
        device = self._where()
        dev = torch.empty(size, dtype=torch.uint8, device=device)
        with torch.cuda.device(device), torch.cuda.stream(torch.cuda.current_stream(device)):
            if capture:
                _lib.check(host.plan_upload(self._plan, -1, dev.data_ptr(), _stream_ptr(None)), "rlt_stage_upload")
            else:
                staging = _PINNED.acquire(size)
                host.plan_arrays(self._plan, staging.buffer.numpy())
                dev.copy_(staging.buffer[:size], non_blocking=True)
                staging.release()
            sent = _Sent(dev, _stream_ptr(None), capture) if dev.is_cuda else None
        base = dev.data_ptr()
        return dev, {name: base + at for name, at in offsets.items()}, sent

    def _arrays_on(self, on: int, capture: int):
        """``_arrays`` for a use on a stream: sent once, on that stream, and once more by each graph that cannot count on that."""
        if self._plan is None:
            return self._arrays[0]
        with self._sending:
            arrays = self._arrays.get(0) or self._arrays.get(capture)
            if arrays is None:
                with _on_stream(on):
                    arrays = self._arrays[capture] = self._send_arrays(capture)
        return arrays

    @contextlib.contextmanager
    def _struct_on(self, stream):
        """The RltBatch for one launch on ``stream``."""
        on = _stream_ptr(stream)
        capture = _lib.load_host().capture(on)
        _, addresses, sent = self._arrays_on(on, capture)
        if sent is not None:
            sent.before(on, capture)
        yield self._struct(addresses)
        if sent is not None:
            sent.after(on, capture)

    def _array_set(self):
        with self._sending if self._plan is not None else contextlib.nullcontext():
            if 0 not in self._arrays:
                self._arrays[0] = self._send_arrays()
        return self._arrays[0]

    @property
    def _dev(self):
        return self._array_set()[0]

    @property
    def _ptr(self):
        return self._array_set()[1]

    @classmethod
    def from_device(cls, src_tables, dst_tables, tok_begin, tok_end, *, block_size: int, exit_planes=None,
                    exit_offsets=None) -> "HandoffBatch":
        """A batch whose arrays already sit in device memory, for instance block tables and exit planes that a peer
        sent over NCCL: nothing is staged, copied or read back. ``src_tables`` / ``dst_tables`` are contiguous int32
        ``[requests, planes, width]`` (either may be None), ``tok_begin`` / ``tok_end`` int32 ``[requests]``,
        ``exit_planes`` int32 with one entry per token and ``exit_offsets`` int64 ``[requests]``. No host-side
        validation is possible; the kernels check ranges, block ids and exit planes and report through the status words.
        """
        tables = src_tables if src_tables is not None else dst_tables
        if tables is None or tables.dim() != 3:
            raise ValueError("block tables must be [requests, planes, width]")
        n, _, width = tables.shape
        if not 1 <= n <= _lib.MAX_REQUESTS:
            raise ValueError(f"a handoff batch holds 1 to {_lib.MAX_REQUESTS} requests")
        checks = [(src_tables, torch.int32, "src_tables"), (dst_tables, torch.int32, "dst_tables"),
                  (tok_begin, torch.int32, "tok_begin"), (tok_end, torch.int32, "tok_end"),
                  (exit_planes, torch.int32, "exit_planes"), (exit_offsets, torch.int64, "exit_offsets")]
        for t, dtype, name in checks:
            if t is not None and (not t.is_cuda or t.dtype != dtype or not t.is_contiguous()):
                raise ValueError(f"{name} must be a contiguous CUDA {dtype} tensor")
        if src_tables is not None and dst_tables is not None and (src_tables.shape[0] != n or dst_tables.shape[0] != n or
                                                                  src_tables.shape[2] != dst_tables.shape[2]):
            raise ValueError("source and destination tables must agree in requests and width")
        if tok_begin.numel() != n or tok_end.numel() != n:
            raise ValueError("one token range per request is required")
        if (exit_planes is None) != (exit_offsets is None) or (exit_offsets is not None and exit_offsets.numel() != n):
            raise ValueError("exit_planes and exit_offsets come as a pair, one offset per request")
        self = cls.__new__(cls)
        self.num_requests, self.table_width, self.block_size = n, width, block_size
        self.ranges, self.total_tokens = None, None
        self.src_planes = src_tables.shape[1] if src_tables is not None else 0
        self.dst_planes = dst_tables.shape[1] if dst_tables is not None else 0
        self.metadata_bytes = 0
        arrays = (src_tables, dst_tables, tok_begin, tok_end, exit_planes, exit_offsets)  # kept alive with the batch
        names = ("src_tables", "dst_tables", "tok_begin", "tok_end", "exit_planes", "exit_offsets")
        self._plan = None
        self._arrays = {0: (arrays, {name: t.data_ptr() for name, t in zip(names, arrays) if t is not None}, None)}
        self.has_exit = exit_planes is not None
        self.exit_count = exit_planes.numel() if exit_planes is not None else 0
        return self

    def as_struct(self) -> _lib.RltBatch:
        """The RltBatch for launches on the current stream."""
        on = _stream_ptr(None)
        return self._struct(self._arrays_on(on, _lib.load_host().capture(on))[1])

    def _struct(self, addresses) -> _lib.RltBatch:
        g = addresses.get
        return _lib.RltBatch(
            self.num_requests, self.table_width, g("src_tables"), g("dst_tables"),
            g("tok_begin"), g("tok_end"), g("exit_planes"), g("exit_offsets"), self.exit_count,
        )


def new_status(device=None) -> torch.Tensor:
    """A zeroed int32 status word array the kernels report data errors into."""
    return torch.zeros(_lib.STATUS_WORDS, dtype=torch.int32, device=device or "cuda")


_STATUS_TEXT = {
    _lib.STATUS_BAD_RANGE: "KV range exceeds allocation",
    _lib.STATUS_BAD_BLOCK: "physical block outside registered pool",
    _lib.STATUS_BAD_PLANE: "exit plane outside the pool's planes",
    _lib.STATUS_TIMEOUT: "timed out waiting for the peer's completion flag",
    _lib.STATUS_STALL: "a bulk copy did not complete within the wait limit",
}


def raise_for_status(status: torch.Tensor) -> None:
    """Synchronising read of a status array; raises like the reference's planner would have."""
    words = status.tolist()
    if words[0] == _lib.STATUS_OK:
        return
    text = _STATUS_TEXT.get(words[0], f"device status {words[0]}")
    if words[0] == _lib.STATUS_STALL:
        raise RuntimeError(f"{text} (CTA {words[1]}, warp {words[2]})")
    if words[0] == _lib.STATUS_TIMEOUT:
        raise TimeoutError(f"{text} (last value {words[1]})")
    raise ValueError(f"{text} (request {words[1]}, detail {words[2]}, {words[3]})")


def _options(mode, layer_begin, layer_end, wire_planes, status, grid_limit, variant, workspace=None,
             plane_begin=0, plane_end=0, deep_layer_mask=0) -> _lib.RltOptions:
    if workspace is not None and (workspace.dtype != torch.uint8 or not workspace.is_contiguous() or not workspace.is_cuda):
        raise ValueError("workspace must be a contiguous CUDA uint8 tensor")
    return _lib.RltOptions(
        int(mode), int(layer_begin), int(layer_end), int(wire_planes),
        status.data_ptr() if status is not None else None, int(grid_limit), int(variant),
        workspace.data_ptr() if workspace is not None else None, workspace.numel() if workspace is not None else 0,
        int(plane_begin), int(plane_end), int(deep_layer_mask),
    )


def dedup_workspace(batch: "HandoffBatch", planes: int, device=None) -> torch.Tensor:
    """Scratch tensor for pack/scatter in ``MODE_DEDUP`` (holds the wire plan of the batch)."""
    n = _lib.load().rlt_kv_dedup_workspace_bytes(batch.num_requests, batch.table_width, planes)
    if n < 0:
        _lib.check(int(n), "rlt_kv_dedup_workspace_bytes")
    return torch.empty(int(n), dtype=torch.uint8, device=device or "cuda")


def dedup_wire_tokens(workspace: torch.Tensor) -> int:
    """(token, plane) pairs on the wire of the last dedup pack/scatter that used ``workspace`` (synchronises)."""
    return int(workspace[:8].view(torch.int64).item())


# --------------------------------------------------------------------------- ops


def kv_handoff(src: PoolView, dst: PoolView, batch: HandoffBatch, *, mode=MODE_ALL_PLANES,
               layer_begin=0, layer_end=0, plane_begin=0, plane_end=0, deep_layers=None, status=None, stream=None,
               grid_limit=0, variant=0) -> None:
    """Pool-to-pool handoff of a batch, straight from source blocks to destination blocks.

    ``layer_begin/layer_end`` and ``plane_begin/plane_end`` restrict the launch to a slice of layers and
    destination planes (0, 0 = everything), which is what layer-by-layer streaming uses. ``deep_layers`` lists
    the layers carried for planes >= 1 (a recurrent-depth model's recurrent layers); plane 0 carries them all.
    """
    mask = 0
    if deep_layers is not None:
        for layer in deep_layers:
            if not 0 <= layer < min(src.num_layers, 64):
                raise ValueError("recurrent_layers must be valid cache layer indices")
            mask |= 1 << layer
        if mask == 0:
            raise ValueError("recurrent_layers must be nonempty and unique")
    rc = batch._move(_lib.MOVE_DIRECT, src, dst, mode=mode, layer_begin=layer_begin, layer_end=layer_end, plane_begin=plane_begin,
                     plane_end=plane_end, mask=mask, status=status, grid_limit=grid_limit, variant=variant, stream=stream)
    if rc != _lib.MOVE_UNSUITED:
        return _lib.check(rc, "rlt_kv_handoff")
    lib = _lib.load()
    s, d = src.as_struct(), dst.as_struct()
    o = _options(mode, layer_begin, layer_end, 0, status, grid_limit, variant, None, plane_begin, plane_end, mask)
    with batch._struct_on(stream) as b:
        _lib.check(lib.rlt_kv_handoff(C.byref(s), C.byref(d), C.byref(b), C.byref(o), _stream_ptr(stream)), "rlt_kv_handoff")


def host_batch_limit() -> int:
    """Largest sum of table and range bytes ``kv_handoff_host`` accepts."""
    return int(_lib.load().rlt_kv_host_batch_limit())


def kv_handoff_host(src: PoolView, dst: PoolView, src_tables: np.ndarray, dst_tables: np.ndarray, tok_begin: np.ndarray,
                    tok_end: np.ndarray, *, layer_begin=0, layer_end=0, plane_begin=0, plane_end=0, status=None,
                    stream=None) -> None:
    """All-planes handoff of a small batch whose tables are host arrays: the library stages them in a slot of its own
    and queues copy and launch on ``stream`` (``rlt_kv_handoff_host``); the arrays are free again on return.

    ``src_tables`` / ``dst_tables`` are C-contiguous int32 ``[requests, planes, width]`` of one width, ``tok_begin`` /
    ``tok_end`` int32 ``[requests]``. Nothing is validated on the host beyond shapes; the kernel checks block ids and
    ranges and reports through ``status``. Raises ``ValueError`` with the library's limit message when the batch does
    not fit a staging slot."""
    _lib.check(_lib.load_host().handoff_host(src._address(), dst._address(), src_tables, dst_tables, tok_begin, tok_end,
                                             layer_begin, layer_end, plane_begin, plane_end, status, _raw_stream(stream)),
               "rlt_kv_handoff_host")


def packed_bytes(pool: PoolView, total_tokens: int, wire_planes: int, layers: int | None = None) -> int:
    lib = _lib.load()
    s = pool.as_struct()
    n = lib.rlt_kv_packed_bytes(C.byref(s), total_tokens, wire_planes, pool.num_layers if layers is None else layers)
    if n < 0:
        _lib.check(int(n), "rlt_kv_packed_bytes")
    return int(n)


def kv_pack(src: PoolView, batch: HandoffBatch, out: torch.Tensor, *, mode=MODE_ALL_PLANES, layer_begin=0,
            layer_end=0, wire_planes=0, status=None, stream=None, grid_limit=0, variant=0, workspace=None) -> None:
    """Gather a batch into ``out`` (uint8, contiguous) in the reference's segment order."""
    if out.dtype != torch.uint8 or not out.is_contiguous() or not out.is_cuda:
        raise ValueError("packed buffer must be a contiguous CUDA uint8 tensor")
    kv_pack_to(src, batch, out.data_ptr(), out.numel(), mode=mode, layer_begin=layer_begin, layer_end=layer_end,
               wire_planes=wire_planes, status=status, stream=stream, grid_limit=grid_limit, variant=variant, workspace=workspace)


def kv_pack_to(src: PoolView, batch: HandoffBatch, out_ptr: int, out_bytes: int, *, mode=MODE_ALL_PLANES, layer_begin=0,
               layer_end=0, wire_planes=0, status=None, stream=None, grid_limit=0, variant=0, workspace=None) -> None:
    """``kv_pack`` into raw memory, typically a staging buffer on the decode GPU mapped through a peer pointer:
    the gather and the push over NVLink become one kernel and nothing is staged on the prefill side."""
    rc = batch._move(_lib.MOVE_PACK, src, None, mode=mode, layer_begin=layer_begin, layer_end=layer_end, wire_planes=wire_planes,
                     status=status, grid_limit=grid_limit, variant=variant, workspace=workspace, packed=out_ptr,
                     packed_bytes=out_bytes, stream=stream)
    if rc != _lib.MOVE_UNSUITED:
        return _lib.check(rc, "rlt_kv_pack")
    lib = _lib.load()
    s = src.as_struct()
    o = _options(mode, layer_begin, layer_end, wire_planes, status, grid_limit, variant, workspace)
    with batch._struct_on(stream) as b:
        _lib.check(lib.rlt_kv_pack(C.byref(s), C.byref(b), C.byref(o), out_ptr, out_bytes, _stream_ptr(stream)), "rlt_kv_pack")


def kv_scatter(packed: torch.Tensor, dst: PoolView, batch: HandoffBatch, *, mode=MODE_ALL_PLANES, layer_begin=0,
               layer_end=0, wire_planes=0, status=None, stream=None, grid_limit=0, variant=0, workspace=None) -> None:
    """Write a packed image into the destination blocks of a batch."""
    if packed.dtype != torch.uint8 or not packed.is_contiguous() or not packed.is_cuda:
        raise ValueError("packed buffer must be a contiguous CUDA uint8 tensor")
    mode = mode if mode == MODE_DEDUP else MODE_ALL_PLANES
    rc = batch._move(_lib.MOVE_SCATTER, None, dst, mode=mode, layer_begin=layer_begin, layer_end=layer_end,
                     wire_planes=wire_planes, status=status, grid_limit=grid_limit, variant=variant, workspace=workspace,
                     packed=packed.data_ptr(), packed_bytes=packed.numel(), stream=stream)
    if rc != _lib.MOVE_UNSUITED:
        return _lib.check(rc, "rlt_kv_scatter")
    lib = _lib.load()
    d = dst.as_struct()
    o = _options(mode, layer_begin, layer_end, wire_planes, status, grid_limit, variant, workspace)
    with batch._struct_on(stream) as b:
        _lib.check(lib.rlt_kv_scatter(packed.data_ptr(), packed.numel(), C.byref(d), C.byref(b), C.byref(o), _stream_ptr(stream)),
                   "rlt_kv_scatter")


def kv_finalize(pool: PoolView, tables: torch.Tensor, rows: torch.Tensor, *, layers=None, status=None, stream=None) -> None:
    """Copy each row's exit-plane K/V (and scales) into every deeper plane.

    ``tables`` is the pool's device ``int32 [requests, planes, width]``; ``rows`` is a device
    ``int32 [n, 3]`` of (request index, exit plane, token position); ``layers`` lists the layers to
    copy (default all; pass the model's recurrent layers for boundary-KV models). For scale tensors
    to be copied the view must carry them: build it with ``PoolView.from_tensors(..., key_scale,
    value_scale)`` also for a fixed-scale pool.
    """
    mask = 0
    if layers is not None:
        for layer in layers:
            if not 0 <= layer < pool.num_layers:
                raise ValueError("recurrent_layers must be valid cache layer indices")
            mask |= 1 << layer
        if mask == 0:
            raise ValueError("recurrent_layers must be nonempty and unique")
    _lib.check(_lib.load_host().finalize(pool._address(), pool.num_planes, tables, rows, mask, status, _raw_stream(stream)),
               "rlt_kv_finalize")


def kv_push(src_ptr: int, dst_ptr: int, nbytes: int, *, stream=None) -> None:
    """Copy one byte range; ``dst_ptr`` may be a peer mapping."""
    _lib.check(_lib.load().rlt_kv_push(src_ptr, dst_ptr, nbytes, _stream_ptr(stream)), "rlt_kv_push")


def kv_copy_segments(segments: torch.Tensor, *, stream=None) -> None:
    """Copy ``int64 [n, 3]`` (source address, destination address, bytes) triples held on the device."""
    if segments.dtype != torch.int64 or segments.dim() != 2 or segments.shape[1] != 3 or not segments.is_contiguous():
        raise ValueError("segments must be a contiguous int64 [n, 3] tensor")
    if not segments.is_cuda:
        raise ValueError("segments must live on the device")
    _lib.check(_lib.load().rlt_kv_copy_segments(segments.data_ptr(), segments.shape[0], _stream_ptr(stream)), "rlt_kv_copy_segments")


def kv_signal(flag_ptr: int, value: int, *, stream=None) -> None:
    _lib.check(_lib.load().rlt_kv_signal(flag_ptr, value, _stream_ptr(stream)), "rlt_kv_signal")


def kv_wait(flag_ptr: int, value: int, timeout_ns: int, status: torch.Tensor, *, stream=None) -> None:
    _lib.check(_lib.load().rlt_kv_wait(flag_ptr, value, timeout_ns, status.data_ptr(), _stream_ptr(stream)), "rlt_kv_wait")


def kernel_launches() -> int:
    return int(_lib.load().rlt_kernel_launches())
