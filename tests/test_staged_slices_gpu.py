"""The slices that staging helpers hand out are ordinary views: writable, of the right place, usable after the array has grown."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64, torch.float32])
def test_an_appended_slice_can_be_changed_until_the_upload(dtype):
    from vllm_rlt_b200.worker.staging import StagedInputTensor

    staged = StagedInputTensor(dtype, "cuda")
    numbers = (lambda *v: [float(x) for x in v]) if dtype.is_floating_point else (lambda *v: list(v))
    staged.append(numbers(*range(8)))
    piece = staged.append(numbers(40, 41, 42))
    assert piece.tolist() == numbers(40, 41, 42) and piece.is_contiguous() and not piece.requires_grad
    piece[1] = 7
    piece.add_(1)
    assert (piece * 2).tolist() == numbers(82, 16, 86)
    sent = staged.upload()
    assert sent.tolist() == numbers(*range(8), 41, 8, 43) and sent.is_cuda
    view = sent[2:4]
    view.zero_()
    assert sent.tolist()[2:4] == numbers(0, 0)


def test_staged_rows_reach_the_middle_of_a_strided_table():
    from vllm_rlt_b200.worker.staging import StagedWriteTensor

    table = torch.zeros(6, 20, dtype=torch.int32, device="cuda")[1:5, 3:17]
    writer = StagedWriteTensor(table, 2, 4)
    writer.stage_write(0, 0, [1, 2])
    writer.stage_write(-1, 11, [3, 4, 5])
    writer.stage_write(2, 13, [6])
    writer.submit()
    want = torch.zeros(4, 14, dtype=torch.int32)
    want[0, :2], want[3, 11:], want[2, 13] = torch.tensor([1, 2]), torch.tensor([3, 4, 5]), 6
    assert torch.equal(table.cpu(), want) and int(table._base.sum()) == 21
    with pytest.raises(ValueError, match="outside the target row"):
        writer.stage_write(0, 13, [1, 2])
