"""Finalize where its split can go wrong: groups that are not full, rows of several requests in one group, rows that need no
copy between rows that do, more planes than one chunk of lookups, narrow rows, a layer subset."""

import random

import numpy as np
import pytest
import torch

from tests.conftest import oracle_pool
from tests.gpu_support import GpuPool, assert_pools_equal
from tests.test_finalize_gpu import full_view

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind, shape, rows", [
    ("bf16", (24, 16, 128, 16, 4), 1), ("bf16", (24, 16, 128, 16, 4), 17), ("fp8", (5, 3, 20, 7, 3), 40),
    ("f32", (2, 1, 3, 4, 2), 33), ("fp8_fixed", (3, 1, 5, 1, 9), 31), ("bf16", (2, 1, 8, 4, 130), 16), ("bf16", (1, 16, 1024, 2, 5), 18),
])
def test_finalize_at_the_edges_of_its_groups(kind, shape, rows):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    layers, heads, dim, page, planes = shape
    rng = random.Random(rows + planes)
    lengths = [rng.randint(1, 2 * page) for _ in range(rows)]
    P = oracle_pool(kind, (layers, heads, dim, sum(-(-n // page) for n in lengths) * planes + 1, page, planes))
    P.fill_random(np.random.default_rng(rows))
    P.shuffle_free_list(rng)
    tables, todo = np.zeros((rows, planes, 2), np.int32), []
    for i, n in enumerate(lengths):
        assert P.allocate(f"r{i}", n)
        for p, t in enumerate(P.plane_block_tables(f"r{i}")):
            tables[i, p, : len(t)] = t
        todo.append((i, rng.choice([0, planes - 1, rng.randrange(planes)]), rng.randrange(n)))
    gp = GpuPool(P)
    for i, e, pos in todo:
        P.finalize_token(f"r{i}", pos, e)
    status = kh.new_status()
    kh.kv_finalize(full_view(gp), torch.from_numpy(tables).cuda(), torch.tensor(todo, dtype=torch.int32, device="cuda"), status=status)
    kh.raise_for_status(status)
    assert_pools_equal(gp, P)


def test_rows_beyond_one_launch_are_served_and_reported_by_their_place_in_the_list():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    one_launch = 1 << 28
    if torch.cuda.mem_get_info()[0] < 5 << 30:
        pytest.skip("needs 5 GiB of free device memory")
    key, value = (torch.randn(6, 1, 4, 1, 16, device="cuda").to(torch.bfloat16) for _ in range(2))
    want = [t.clone() for t in (key, value)]
    rows = torch.empty(one_launch + 5, 3, dtype=torch.int32, device="cuda")
    rows[:] = torch.tensor([0, 1, 0], dtype=torch.int32)  # the deepest plane: nothing to copy
    for at, position in ((0, 0), (one_launch - 1, 5), (one_launch, 2), (one_launch + 4, 7)):
        rows[at, 1], rows[at, 2] = 0, position
        for t in want:
            t[3 + position // 4, 0, position % 4] = t[1 - position // 4, 0, position % 4]
    rows[one_launch + 2, 1] = 2  # no such plane
    tables = torch.tensor([[[1, 0], [3, 4]]], dtype=torch.int32, device="cuda")
    status = kh.new_status()
    before = kh.kernel_launches()
    kh.kv_finalize(kh.PoolView.from_tensors(key, value, 2), tables, rows, status=status)
    assert status.tolist() == [3, one_launch + 2, 0, 2] and kh.kernel_launches() == before + 2
    assert torch.equal(key, want[0]) and torch.equal(value, want[1])


def test_a_layer_past_the_ones_that_can_be_selected_is_refused_in_words():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    cache = torch.zeros(2, 70, 4, 1, 16, dtype=torch.bfloat16, device="cuda")
    tables = torch.zeros(1, 2, 1, dtype=torch.int32, device="cuda")
    rows = torch.zeros(1, 3, dtype=torch.int32, device="cuda")
    for layers in ([69], [64], None):
        with pytest.raises(ValueError, match="limit"):
            kh.kv_finalize(kh.PoolView.from_tensors(cache, cache.clone(), 2), tables, rows, layers=layers)
