"""The flat copy around its vectors: heads, tails, sizes below one vector, tensors that are aligned together, apart or never."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("types", [(torch.int64, torch.int32, None), (torch.bfloat16, torch.bfloat16, None),
                                   (torch.float16, torch.int64, torch.bfloat16), (torch.float32, torch.float16, torch.int32)])
@pytest.mark.parametrize("n", [1, 7, 8, 31, 33, 2047, 4096, 4097, 40001])
@pytest.mark.parametrize("skips", [(0, 0), (1, 1), (3, 3), (1, 0), (15, 15)])
def test_flat_copies_of_any_start_and_length(types, n, skips):
    from vllm_rlt_b200.worker.tensors import copy_tensor

    source_type, target_type, second_type = types
    source = (torch.arange(n + 16, device="cuda") % 2000).to(source_type)[skips[0] : skips[0] + n]
    target = torch.full((n + 40,), 99, device="cuda").to(target_type)
    second = None if second_type is None else torch.full((n + 40,), 99, device="cuda").to(second_type)
    cut = slice(skips[1], skips[1] + n)
    copy_tensor(source, target[cut], secondary=None if second is None else second[cut])
    for out in (target, second) if second is not None else (target,):
        assert torch.equal(out[cut], source.to(out.dtype))
        assert bool((out[: skips[1]] == 99).all()) and bool((out[skips[1] + n :] == 99).all())
