"""Several threads and streams at once: a call that has to wait for the GPU holds up neither the threads that need not wait nor the
one whose word the GPU is waiting for. Every wait on the GPU is bounded (``kv_wait``) and ends when the host sets its flag."""

import ctypes as C
import threading
import time

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LIMIT_NS = 2_000_000_000  # of the waits on the GPU; a test that passes sets their flags long before
PAGES = 1000              # 8 words a page: more than the kernel parameters hold, and one staging slot


class Waiting:
    """A stream whose work, from now on, waits until the host says ``go``."""

    def __init__(self, stream=None):
        from vllm_rlt_b200.kernels import kv_handoff as kh

        self.flag = torch.zeros(1, dtype=torch.int64, pin_memory=True)
        self.status = kh.new_status()
        self.stream = stream or torch.cuda.Stream()
        self.stream.wait_stream(torch.cuda.current_stream())
        kh.kv_wait(self.flag.data_ptr(), 1, LIMIT_NS, self.status, stream=self.stream)

    def go(self):
        self.flag[0] = 1

    def in_time(self):
        self.stream.synchronize()
        return self.status.tolist() == [0, 0, 0, 0]


@pytest.fixture(scope="module")
def pools():
    """Two single-plane pools of PAGES + 1 blocks and tables over PAGES of them."""
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.kernels import kv_handoff as kh

    src, dst = (KVPool(1, 1, 16, PAGES + 1, 4, 1, device="cuda") for _ in range(2))
    src.key_cache.normal_()
    src.value_cache.normal_()
    tables = np.random.default_rng(0).permutation(PAGES).astype(np.int32).reshape(1, 1, PAGES)
    return src, dst, kh.PoolView.from_cache(src), kh.PoolView.from_cache(dst), tables


def arrived(pools):
    src, dst, _, _, tables = pools
    at = torch.from_numpy(tables.reshape(-1)).cuda().long()
    whole = all(torch.equal(a[at], b[at]) for a, b in ((src.key_cache, dst.key_cache), (src.value_cache, dst.value_cache)))
    for t in (dst.key_cache, dst.value_cache):
        t.zero_()
    return whole


def test_a_call_that_finds_a_free_slot_is_not_held_up_by_one_that_waits_for_its_own(pools):
    from vllm_rlt_b200 import _lib

    _, _, sv, dv, tables = pools
    lib = _lib.load()  # through ctypes, which lets other threads run
    s, d = sv.as_struct(), dv.as_struct()
    begin, end = np.zeros(1, np.int32), np.full(1, 4 * PAGES, np.int32)
    batch = _lib.RltHostBatch(1, PAGES, 1, 1, tables.ctypes.data, tables.ctypes.data, begin.ctypes.data, end.ctypes.data)
    options = _lib.RltOptions()
    device = torch.cuda.current_device()

    def call(stream):
        torch.cuda.set_device(device)
        _lib.check(lib.rlt_kv_handoff_host(C.byref(s), C.byref(d), C.byref(batch), C.byref(options), stream.cuda_stream), "handoff")

    call(torch.cuda.current_stream())
    torch.cuda.synchronize()
    a, b = Waiting(), Waiting()
    for w in (a, b):
        for _ in range(8):  # all 16 slots of the library
            call(w.stream)
    late = threading.Thread(target=call, args=(a.stream,))
    late.start()
    time.sleep(0.1)
    assert late.is_alive()  # it waits for a slot of stream a's launches
    b.go()
    b.stream.synchronize()
    began = time.monotonic()
    call(b.stream)
    took = time.monotonic() - began
    a.go()
    late.join(timeout=10)
    assert not late.is_alive() and took < 0.5
    assert a.in_time() and b.in_time() and arrived(pools)


def test_a_batch_whose_image_another_thread_lays_out_for_other_planes_packs_its_own(monkeypatch):
    """Between a pack's look at the layout of its image and its launch another thread may use the same batch for an image of another
    plane count. (Here the launch itself lets that happen, at the one point where it matters.)"""
    import random

    from oracle import handoff_oracle as ho
    from tests.conftest import oracle_pool
    from tests.gpu_support import GpuPool
    from vllm_rlt_b200.kernels import kv_handoff as kh

    planes, page, lengths = 4, 4, [30, 11]
    P = oracle_pool("bf16", (2, 1, 16, 64, page, planes))
    P.fill_random(np.random.default_rng(3))
    rng, exits = random.Random(3), []
    for i, n in enumerate(lengths):
        assert P.allocate(f"r{i}", n)
        exits.append([rng.randrange(planes) for _ in range(n)])
    tables = [P.plane_block_tables(f"r{i}") for i in range(len(lengths))]
    want = np.concatenate([ho.pack_rows(P, t, 0, n, mode=ho.MODE_DEDUP, exit_planes=e) for t, n, e in zip(tables, lengths, exits)])
    gp = GpuPool(P)
    batch = kh.HandoffBatch(tables, None, [(0, n) for n in lengths], block_size=page, exit_planes=exits)
    workspace, status = kh.dedup_workspace(batch, planes), kh.new_status()
    packed = torch.zeros(kh.packed_bytes(gp.view(), batch.total_tokens, planes), dtype=torch.uint8, device="cuda")
    host = kh._lib.load_host()

    class Interrupted:
        def __getattr__(self, name):
            return getattr(host, name)

        def move(self, *arguments):
            host.plan_wire(batch._plan, 2)
            return host.move(*arguments)

    monkeypatch.setattr(kh._lib, "load_host", Interrupted)
    kh.kv_pack(gp.view(), batch, packed, mode=kh.MODE_DEDUP, status=status, workspace=workspace)
    kh.raise_for_status(status)
    assert np.array_equal(packed.cpu().numpy()[: want.size], want)
    assert kh.dedup_wire_tokens(workspace) == sum(e + 1 for row in exits for e in row)


@pytest.mark.parametrize("what", ["host tables", "batch records", "transport tables"])
def test_the_thread_that_the_gpu_waits_for_runs_while_another_waits_for_the_gpu(pools, what):
    """More calls than there are staging slots, on a stream that waits for a word another Python thread writes: the calls wait for a
    slot, and that thread has to get the interpreter meanwhile."""
    from vllm_rlt_b200 import _lib
    from vllm_rlt_b200.kernels import kv_handoff as kh

    _, _, sv, dv, tables = pools
    begin, end = np.zeros(1, np.int32), np.full(1, 4 * PAGES, np.int32)
    w = Waiting()
    keep = []

    def call():
        if what == "host tables":
            kh.kv_handoff_host(sv, dv, tables, tables, begin, end, stream=w.stream)
        elif what == "transport tables":
            side = (tables[0, 0],)
            _lib.check(_lib.load_host().handoff_requests(sv._address(), dv._address(), [(side, side, 0, 4 * PAGES)], 0, 0, 0, 0, 0,
                                                         w.stream.cuda_stream), "handoff")
        else:
            keep.append(kh.HandoffBatch(tables, tables, [(0, 4 * PAGES)], block_size=4, stream=w.stream))

    def release():
        time.sleep(0.3)
        w.go()

    other = threading.Thread(target=release)
    other.start()
    began = time.monotonic()
    for _ in range(70 if what == "batch records" else 20):
        call()
    took = time.monotonic() - began
    other.join(timeout=10)
    assert w.in_time() and took > 0.2  # the calls did have to wait
    if what == "batch records":
        kh.kv_handoff(sv, dv, keep[-1], stream=w.stream)
        w.stream.synchronize()
    assert arrived(pools)


def test_copies_appended_while_another_thread_submits_do_not_disturb_the_submission():
    from vllm_rlt_b200.worker.tensors import TensorTransfer

    rows = 256
    source = torch.arange(rows * 64, dtype=torch.int32, device="cuda").reshape(rows, 64)
    target = torch.zeros_like(source)
    mover = TensorTransfer(4096, torch.int32, "cuda:0")
    for i in range(rows):
        mover.append(source[i], target[i])
    torch.cuda.synchronize()
    stop, wrong = threading.Event(), []

    def submitting():
        torch.cuda.set_device(0)
        while not stop.is_set():
            mover.submit()
            if not stop.is_set() and mover.max_cols != 64:
                wrong.append(mover.max_cols)

    thread = threading.Thread(target=submitting)
    thread.start()
    for _ in range(2000):
        mover.append(source[3], target[3])
    stop.set()
    thread.join(timeout=20)
    mover.submit()
    torch.cuda.synchronize()
    assert not thread.is_alive() and not wrong and torch.equal(source, target)


def test_a_batch_used_on_another_stream_waits_for_its_records_and_for_nothing_else(pools):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    _, _, sv, dv, tables = pools
    for variant in (0, 5):  # the records, and the padded arrays of the table-driven kernels
        own, third = torch.cuda.Stream(), torch.cuda.Stream()
        batch = kh.HandoffBatch(tables, tables, [(0, 4 * PAGES)], block_size=4, stream=own)
        if variant:
            kh.kv_handoff(sv, dv, batch, variant=variant, stream=own)
        w = Waiting(own)  # work that has nothing to do with the batch
        for stream in (third, torch.cuda.current_stream()):
            kh.kv_handoff(sv, dv, batch, variant=variant, stream=stream)
            done = stream.record_event()
            began = time.monotonic()
            while not done.query() and time.monotonic() - began < 0.5:
                time.sleep(0.001)
            assert done.query() and arrived(pools)
        w.go()
        assert w.in_time()


@pytest.mark.parametrize("default", [True, False])
def test_a_use_on_any_other_stream_does_wait_for_the_records(pools, default):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    _, _, sv, dv, tables = pools
    w = Waiting()
    batch = kh.HandoffBatch(tables, tables, [(0, 4 * PAGES)], block_size=4, stream=w.stream)  # sent behind the wait
    user = torch.cuda.current_stream() if default else torch.cuda.Stream()
    kh.kv_handoff(sv, dv, batch, stream=user)
    done = user.record_event()
    time.sleep(0.2)
    assert not done.query()
    w.go()
    user.synchronize()
    assert w.in_time() and arrived(pools)


def test_a_batch_that_is_dropped_keeps_its_records_until_every_stream_has_used_them(pools):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    _, _, sv, dv, tables = pools
    own = torch.cuda.Stream()
    batch = kh.HandoffBatch(tables, tables, [(0, 4 * PAGES)], block_size=4, stream=own)
    size = batch.metadata_bytes
    w = Waiting()
    kh.kv_handoff(sv, dv, batch, stream=w.stream)
    del batch
    with torch.cuda.stream(own):
        # the memory's next owner writes it; records of zeros name no token
        others = [torch.zeros(size, dtype=torch.uint8, device="cuda") for _ in range(8)]
    time.sleep(0.1)
    w.go()
    assert w.in_time() and arrived(pools)
    own.synchronize()
    assert not any(bool(t.any()) for t in others)
