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
