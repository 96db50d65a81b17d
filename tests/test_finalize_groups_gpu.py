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
