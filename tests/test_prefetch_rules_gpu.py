"""Which launches ask L2 for their source: those that move 32 MB and more out of this GPU's own memory."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def counted(launch):
    """Launches that asked, and addresses that were looked up for it."""
    from vllm_rlt_b200 import _lib

    before, after = (ctypes.c_int64 * 2)(), (ctypes.c_int64 * 2)()
    _lib.load().rlt_prefetch_counts(before)
    launch()
    _lib.load().rlt_prefetch_counts(after)
    return after[0] - before[0], after[1] - before[1]


def copy(ranges):
    from vllm_rlt_b200 import _lib

    triples = np.array(ranges, np.int64).tobytes()
    return counted(lambda: _lib.check(_lib.load_host().copy_segments(triples, 0, None), "copy"))


def test_pushes_and_flat_copies():
    from vllm_rlt_b200.kernels import kv_handoff as kh
    from vllm_rlt_b200.worker.tensors import copy_tensor

    n = 16 << 20
    a, b = (torch.zeros(n + 64, dtype=torch.uint8, device="cuda") for _ in range(2))
    held = torch.ones(n + 64, dtype=torch.uint8, pin_memory=True)
    assert counted(lambda: kh.kv_push(a.data_ptr(), b.data_ptr(), n)) == (1, 1)
    assert counted(lambda: kh.kv_push(a.data_ptr(), b.data_ptr(), n - 1)) == (0, 0)
    assert counted(lambda: kh.kv_push(held.data_ptr(), b.data_ptr(), n)) == (0, 1)
    assert torch.equal(b[:n].cpu(), held[:n])
    x, y = a.view(torch.int32), b.view(torch.int32)
    assert counted(lambda: copy_tensor(x[: n // 4], y[: n // 4])) == (1, 1)
    assert counted(lambda: copy_tensor(x[: n // 4], y[1 : n // 4 + 1])) == (0, 0)  # element by element
    torch.cuda.synchronize()


@pytest.mark.parametrize("count, size, asks", [(1024, 33, False), (1024, (16 << 10) - 1, False), (1024, 16 << 10, True), (171, 100_000, True),
                                               (1, 16 << 20, True), (1, (16 << 20) - 1, False)])
def test_lists_count_the_bytes_that_they_move(count, size, asks):
    a, b = (torch.randint(0, 256, (count * size,), dtype=torch.uint8, device="cuda") for _ in range(2))
    got = copy([(a.data_ptr() + i * size, b.data_ptr() + i * size, size) for i in range(count)])
    assert got == ((1, 1) if asks else (0, 0))
    assert torch.equal(a, b)


def test_lists_with_other_memory_among_their_sources_do_not_ask():
    n = 8 << 20
    mine = [torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda") for _ in range(3)]
    held = torch.randint(0, 256, (n,), dtype=torch.uint8).pin_memory()
    out = torch.zeros(4 * n, dtype=torch.uint8, device="cuda")
    for at in range(4):  # first, among the others, last
        sources = mine[:at] + [held] + mine[at:]
        asked, looked = copy([(s.data_ptr(), out.data_ptr() + i * n, n) for i, s in enumerate(sources)])
        assert asked == 0 and 1 <= looked <= at + 1  # tensors may share an allocation
        assert torch.equal(out, torch.cat([s.cuda() for s in sources]))
    asked, looked = copy([(s.data_ptr(), out.data_ptr() + i * n, n) for i, s in enumerate(mine)])
    assert asked == 1 and 1 <= looked <= 3


def test_lists_over_many_allocations():
    """As many tensors as a worker's pools have, and the rows beside them, are asked for; ranges all over the place are not."""
    size = 20 << 20  # each an allocation of its own
    parts = [torch.randint(0, 256, (size,), dtype=torch.uint8, device="cuda") for _ in range(12)]
    out = torch.zeros(12 * size, dtype=torch.uint8, device="cuda")
    bases = len({p.untyped_storage().data_ptr() for p in parts})
    assert bases == 12
    for tensors in (4, 5, 12):
        ranges = [(p.data_ptr() + k * 4096, out.data_ptr() + i * size + k * 4096, 4096) for k in range(80) for i, p in enumerate(parts[:tensors])]
        ranges += [(p.data_ptr() + 80 * 4096, out.data_ptr() + i * size + 80 * 4096, size - 80 * 4096) for i, p in enumerate(parts[:tensors])]
        asked, looked = copy(ranges)
        assert looked <= 8 and (asked == 1 or tensors == 12)
    assert torch.equal(out, torch.cat(parts))


def handoff(pages, planes, mode, *, layers=24, heads=16, dim=128, page=16, tokens=None, fp8=False):
    """A handoff of one request of so many pages, counted."""
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.kernels import kv_handoff as kh

    kind = "fp8_e4m3" if fp8 else "auto"
    src = KVPool(layers, heads, dim, pages * planes, page, planes, kv_cache_dtype=kind)
    to = 1 if mode == kh.MODE_EXIT_ONLY else planes
    dst = KVPool(layers, heads, dim, pages * to, page, to, kv_cache_dtype=kind)
    for t in (src.key_cache, src.value_cache):
        t.view(torch.uint8).random_(0, 255)
    tokens = pages * page if tokens is None else tokens
    st = [np.arange(p * pages, (p + 1) * pages, dtype=np.int32) for p in range(planes)]
    dt = [np.arange(p * pages, (p + 1) * pages, dtype=np.int32) for p in range(to)]
    exits = None if mode == kh.MODE_ALL_PLANES else [np.arange(tokens, dtype=np.int32) % planes]
    batch = kh.HandoffBatch([st], [dt], [(0, tokens)], block_size=page, exit_planes=exits)
    got = counted(lambda: kh.kv_handoff(kh.PoolView.from_cache(src), kh.PoolView.from_cache(dst), batch, mode=mode))
    if mode == kh.MODE_ALL_PLANES and tokens == pages * page:
        for a, b in ((src.key_cache, dst.key_cache), (src.value_cache, dst.value_cache)):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    torch.cuda.synchronize()
    return got, bool(batch._staged)


def test_handoffs_ask_while_their_records_are_parameters():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    assert handoff(20, 4, kh.MODE_ALL_PLANES) == ((1, 2), False)
    assert handoff(1, 4, kh.MODE_ALL_PLANES) == ((0, 0), False)  # 25 MB
    assert handoff(20, 4, kh.MODE_ALL_PLANES, fp8=True, layers=48)[0] == (1, 4)  # codes and scales
    assert handoff(20, 2, kh.MODE_ALL_PLANES, fp8=True, layers=48, heads=3, dim=256)[0] == (1, 2)  # rows of 12 bytes are not asked for
    got, staged = handoff(600, 4, kh.MODE_ALL_PLANES)  # records of 33 KB: in device memory, where nothing can be asked for
    assert staged and got == (0, 0)
    assert handoff(40, 4, kh.MODE_EXIT_ONLY)[0] == (1, 2)
    assert handoff(300, 4, kh.MODE_EXIT_ONLY)[0] == (0, 0)  # records too large
    assert handoff(40, 4, kh.MODE_DEDUP)[0] == (0, 0)  # no kind that asks


def test_pages_that_are_mostly_not_full_are_not_asked_for():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    assert handoff(1, 12, kh.MODE_ALL_PLANES, page=64, tokens=47)[0] == (0, 0)
    assert handoff(1, 12, kh.MODE_ALL_PLANES, page=64, tokens=48)[0] == (1, 2)
    assert handoff(2, 12, kh.MODE_ALL_PLANES, page=64, tokens=65)[0] == (0, 0)  # every second one is whole
    assert handoff(2, 12, kh.MODE_ALL_PLANES, page=64, tokens=96)[0] == (1, 2)


def test_pool_tensors_elsewhere():
    """Keys in this GPU's memory and values in pinned memory: nothing is asked for, and both arrive."""
    from vllm_rlt_b200 import _lib
    from vllm_rlt_b200.kernels import kv_handoff as kh

    shape = (8, 24, 16, 16, 128)
    key = torch.randint(-100, 100, shape, dtype=torch.int16, device="cuda")
    value = torch.randint(-100, 100, shape, dtype=torch.int16).pin_memory()
    out = [torch.zeros(shape, dtype=torch.int16, device="cuda") for _ in range(2)]
    token = 16 * 128 * 2

    def pool(k, v):
        region = _lib.RltRegion(k.data_ptr(), v.data_ptr(), 24 * 16 * token, 16 * token, token)
        return _lib.RltPool(region, _lib.RltRegion(), 8, 16, 24, 1)

    tables = np.arange(8, dtype=np.int32)
    begin, end = np.zeros(1, np.int32), np.array([128], np.int32)
    hb = _lib.RltHostBatch(1, 8, 1, 1, tables.ctypes.data, tables.ctypes.data, begin.ctypes.data, end.ctypes.data)
    stream = torch.cuda.current_stream().cuda_stream

    def launch(src):
        return counted(lambda: _lib.check(_lib.load().rlt_kv_handoff_host(ctypes.byref(src), ctypes.byref(pool(*out)), ctypes.byref(hb),
                                                                          ctypes.byref(_lib.RltOptions()), stream), "handoff"))

    assert launch(pool(key, value)) == (0, 2)
    assert torch.equal(out[0], key) and torch.equal(out[1].cpu(), value)
    assert launch(pool(value, key)) == (0, 1)
    assert torch.equal(out[1], key) and torch.equal(out[0].cpu(), value)
    assert launch(pool(key, key)) == (1, 2)
    assert torch.equal(out[1], key)
