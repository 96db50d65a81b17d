"""Wire images whose rows are at places that the pool's vectors do not fit: FP8 codes beside the scales of a number of heads that is no multiple of
four. Packed images equal the oracle's, and scattering them leaves what the oracle's handoff leaves."""

import random

import numpy as np
import pytest
import torch

from oracle import handoff_oracle as ho
from tests.conftest import oracle_pool
from tests.gpu_support import GpuPool, assert_pools_equal
from tests.test_kv_handoff_gpu import sentinel_destination

pytestmark = pytest.mark.gpu


# (heads, dim): rows on 4-byte boundaries of the image with 16- and 32-byte rows in the pool, on 8-byte ones, on 16-byte ones
@pytest.mark.parametrize("heads, dim", [(1, 16), (3, 32), (5, 48), (2, 64), (6, 16), (4, 32)])
@pytest.mark.parametrize("mode", [ho.MODE_ALL_PLANES, ho.MODE_DEDUP, ho.MODE_EXIT_ONLY])
@pytest.mark.parametrize("page, layers", [(16, 5), (7, 40), (64, 3)])
def test_images_with_rows_at_odd_places(heads, dim, mode, page, layers):
    from vllm_rlt_b200.kernels import kv_handoff as k

    planes, lengths = 3, [1, page, 2 * page + 5, 70]
    rng = random.Random(heads * dim + page)
    shape = (layers, heads, dim, sum(-(-n // page) for n in lengths) * planes + 3, page, planes)
    wire = 1 if mode == ho.MODE_EXIT_ONLY else planes
    P, D = oracle_pool("fp8", shape), sentinel_destination("fp8", shape, planes=wire)
    P.fill_random(np.random.default_rng(dim))
    for pool in (P, D):
        pool.shuffle_free_list(rng)
    ranges, exits = [], []
    for i, n in enumerate(lengths):
        assert P.allocate(f"r{i}", n) and D.allocate(f"r{i}", n)
        ranges.append((min(i, n - 1), n))
        exits.append([rng.randrange(planes) for _ in range(n)])
        for pos in range(n) if mode == ho.MODE_DEDUP else ():
            P.finalize_token(f"r{i}", pos, exits[i][pos])
    src, dst = ([pool.plane_block_tables(f"r{i}") for i in range(len(lengths))] for pool in (P, D))
    gp, gd = GpuPool(P), GpuPool(D)
    batch = k.HandoffBatch(src, dst, ranges, block_size=page, exit_planes=None if mode == ho.MODE_ALL_PLANES else exits)
    status = k.new_status()
    workspace = k.dedup_workspace(batch, planes) if mode == ho.MODE_DEDUP else None
    packed = torch.full((k.packed_bytes(gp.view(), batch.total_tokens, wire) + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    k.kv_pack(gp.view(), batch, packed, mode=mode, status=status, workspace=workspace)
    want = np.concatenate([ho.pack_rows(P, src[i], s, e, mode=mode, exit_planes=exits[i]) for i, (s, e) in enumerate(ranges)])
    got = packed.cpu().numpy()
    assert np.array_equal(got[: want.size], want) and (got[want.size :] == 0x5A).all()
    k.kv_scatter(packed, gd.view(), batch, mode=mode if mode == ho.MODE_DEDUP else 0, status=status, workspace=workspace)
    k.raise_for_status(status)
    for i, (s, e) in enumerate(ranges):
        ho.handoff_rows(P, D, src[i], dst[i], s, e, mode=mode, exit_planes=exits[i])
    assert_pools_equal(gd, D)

    # an image that ends early: what lies behind its end is neither written nor read
    short = want.size - want.size // 3 & ~15
    packed.fill_(0x5A)
    k.kv_pack(gp.view(), batch, packed[:short], mode=mode, status=status, workspace=workspace)
    assert status[0] != 0 and (packed[short:] == 0x5A).all()
