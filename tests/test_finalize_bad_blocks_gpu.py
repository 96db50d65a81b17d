"""Finalize with a block table entry that is no block's, at each place among those that a thread looks up together and one by one."""

import numpy as np
import pytest
import torch

from tests.conftest import oracle_pool
from tests.gpu_support import GpuPool, assert_pools_equal
from tests.test_finalize_gpu import full_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, shape", [("bf16", (3, 2, 16, 24, 4, 6)), ("fp8", (3, 3, 16, 24, 4, 6))])
@pytest.mark.parametrize("exit_plane", [0, 2, 4])
@pytest.mark.parametrize("bad", [(0,), (1,), (2,), (3,), (4,), (5,), (3, 5), (1, 2, 3, 4, 5)])
def test_rows_reach_every_plane_whose_block_is_one(kind, shape, exit_plane, bad):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    P = oracle_pool(kind, shape)
    P.fill_random(np.random.default_rng(sum(bad)))
    assert P.allocate("a", 4)
    gp, before = GpuPool(P), P
    table = [list(t) for t in P.plane_block_tables("a")]
    good = [row[0] for row in table]
    for plane in bad:
        table[plane][0] = shape[3] + plane
    status = kh.new_status()
    kh.kv_finalize(full_view(gp), torch.tensor([table], dtype=torch.int32, device="cuda"),
                   torch.tensor([[0, exit_plane, 1]], dtype=torch.int32, device="cuda"), status=status)
    looked_up = [p for p in bad if p >= exit_plane]
    first = exit_plane if exit_plane in bad else min(looked_up, default=None)
    assert status.tolist() == ([0] * 4 if first is None else [2, 0, 0, shape[3] + first])
    if exit_plane not in bad:
        for plane in range(exit_plane + 1, shape[5]):
            if plane not in bad:
                for t in before.tensors(travelling_only=False):
                    t.data[good[plane], :, 1] = t.data[good[exit_plane], :, 1]
    assert_pools_equal(gp, before)
