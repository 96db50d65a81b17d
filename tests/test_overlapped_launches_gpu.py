"""Launches that are set up while the one before them still runs read what that one leaves behind: payload, descriptor tables and lists of small copies
that are written anew by the launch just ahead, again and again with other values."""

import pytest
import torch

pytestmark = pytest.mark.gpu

TURNS = 200
CODES = {torch.int32: 0, torch.int64: 1, torch.float32: 4}  # the C ABI's


# aligned, past an aligned place by one element (heads), no common alignment (element by element); from one launch's worth to many blocks
@pytest.mark.parametrize("n", [5, 4096, 100_003, 1_500_001])
@pytest.mark.parametrize("source_skip, target_skip", [(0, 0), (1, 1), (1, 0)])
@pytest.mark.parametrize("kinds", [(torch.int64, torch.int32), (torch.int32, torch.int64), (torch.int32, torch.int32), (torch.float32, torch.bfloat16)])
def test_flat_copies_read_what_the_launch_ahead_wrote(n, source_skip, target_skip, kinds):
    from vllm_rlt_b200.worker.tensors import copy_tensor

    source, target = kinds
    values = [torch.randint(0, 256, (n,), device="cuda").to(source) for _ in range(4)]
    between = torch.zeros(n + source_skip, dtype=source, device="cuda")[source_skip:]
    outs = [torch.zeros(n + target_skip, dtype=target, device="cuda")[target_skip:] for _ in values]
    torch.cuda.synchronize()
    for turn in range(TURNS):
        copy_tensor(values[turn % 4], between)
        copy_tensor(between, outs[turn % 4])
    for out, value in zip(outs, values):
        assert torch.equal(out, value.to(target))


@pytest.mark.parametrize("rows, cols", [(1, 1), (3, 700), (9, 4097)])
@pytest.mark.parametrize("kinds", [(torch.int32, torch.int32), (torch.int64, torch.float32)])
def test_descriptor_tables_that_the_launch_ahead_wrote(rows, cols, kinds):
    """The table names another source and another destination each time it is written."""
    from vllm_rlt_b200 import _lib
    from vllm_rlt_b200.worker.tensors import copy_tensor

    source, target = kinds
    fresh = [torch.randint(0, 1 << 20, (2, rows, cols), device="cuda").to(source) for _ in range(5)]
    a = [torch.zeros_like(fresh[0]) for _ in range(3)]
    b = [torch.zeros(2, rows, cols, dtype=target, device="cuda") for _ in a]
    tables = [torch.tensor([[x[k].data_ptr(), y[k].data_ptr(), rows, cols, cols, 1, cols, 1] for k in range(2)], dtype=torch.int64, device="cuda")
              for x, y in zip(a, b)]
    table = tables[0].clone()
    stream = torch.cuda.current_stream().cuda_stream
    torch.cuda.synchronize()
    for turn in range(TURNS):
        k = turn % 3
        copy_tensor(fresh[turn % 5].view(-1), a[k].view(-1))  # the payload too is written just ahead
        copy_tensor(tables[k].view(-1), table.view(-1))
        _lib.check(_lib.load().rlt_tensor_transfer(table.data_ptr(), 2, rows, cols, CODES[source], CODES[target], stream), "transfer")
    for turn in range(TURNS - 3, TURNS):
        assert torch.equal(b[turn % 3], fresh[turn % 5].to(target))


@pytest.mark.parametrize("count, columns", [(1, 1), (7, 300), (96, 2048)])
def test_small_copies_read_what_the_launch_ahead_wrote(count, columns):
    """Rows handed on through a chain of buffers, one launch behind another."""
    from vllm_rlt_b200.worker.tensors import TensorTransfer

    chain = [torch.randint(-1000, 1000, (count, columns), dtype=torch.int16, device="cuda").view(torch.bfloat16)]
    chain += [torch.zeros_like(chain[0]) for _ in range(6)]
    mover = TensorTransfer(count, torch.bfloat16, "cuda:0")
    for turn in range(TURNS // 4):
        chain[0].view(torch.int16).add_(1)
        for here, there in zip(chain, chain[1:]):
            mover.reset()
            for i in range(count):
                mover.append(here[i], there[count - 1 - i])
            mover.submit()
        assert torch.equal(chain[-1].view(torch.int16), chain[0].view(torch.int16))
