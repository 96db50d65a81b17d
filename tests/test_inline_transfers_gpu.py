"""Batches of copies between tensors of one type around the sizes where their descriptors change places (56 and 448 copies) and
where a row changes from vectors to single elements."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.int32, torch.int64])
@pytest.mark.parametrize("count", [1, 56, 57, 448, 449])
@pytest.mark.parametrize("cols", [1, 7, 512, 4104])
def test_many_small_copies_land_exactly(dtype, count, cols):
    from vllm_rlt_b200.worker.tensors import TensorTransfer

    source = torch.arange(6 * (cols + 3), device="cuda").reshape(6, cols + 3).to(dtype)
    target = torch.zeros(count, 5, cols + 9, dtype=dtype, device="cuda")
    want = target.clone()
    batch = TensorTransfer(count, dtype, "cuda:0")
    for i in range(count):
        shift = i % 3  # a source that starts between two vectors
        if i % 2:
            pair = source[i % 6, shift : shift + cols], target[i, 4, 8 : 8 + cols]
            want[i, 4, 8 : 8 + cols] = source[i % 6, shift : shift + cols]
        else:
            pair = source[:5, shift : shift + cols], target[i, :, 1 : 1 + cols]
            want[i, :, 1 : 1 + cols] = source[:5, shift : shift + cols]
        batch.append(*pair)
    batch.submit()
    assert torch.equal(target, want)
