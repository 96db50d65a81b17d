"""The record kernels at the edges of their dispatch, against the oracle: records as small and as large kernel parameters
and in device memory, the most planes and the largest and smallest pages, every vector width, several rounds per CTA."""

import random

import numpy as np
import pytest
import torch

from oracle import handoff_oracle as ho
from tests.conftest import oracle_pool
from tests.gpu_support import GpuPool, assert_pools_equal
from tests.test_kv_handoff_gpu import sentinel_destination

pytestmark = pytest.mark.gpu

# kind, (layers, heads, dim, page, planes), prompt lengths
CASES = {
    "one token": ("bf16", (1, 1, 16, 16, 2), [1]),
    "small parameters, narrow rows": ("f32", (2, 1, 3, 4, 3), [9, 2]),
    "large parameters": ("fp8", (3, 3, 20, 7, 4), [60, 33, 91]),
    "device records": ("bf16", (2, 1, 8, 1, 4), [400, 1, 301]),
    "device records, odd bytes": ("fp8_fixed", (1, 1, 5, 1, 3), [700, 77]),
    "64 planes of 64-token pages": ("bf16", (2, 1, 16, 64, 64), [65, 3]),
    "several rounds": ("bf16", (24, 8, 64, 16, 4), [150, 170]),
}


@pytest.mark.parametrize("mode", [ho.MODE_ALL_PLANES, ho.MODE_DEDUP, ho.MODE_EXIT_ONLY])
@pytest.mark.parametrize("name", CASES)
def test_handoff_pack_and_scatter_from_records_equal_the_oracle(name, mode):
    from vllm_rlt_b200.kernels import kv_handoff as k

    kind, (layers, heads, dim, page, planes), lengths = CASES[name]
    rng = random.Random(10 * len(name) + mode)
    blocks = sum(-(-n // page) for n in lengths) * planes + 3
    dst_planes = 1 if mode == ho.MODE_EXIT_ONLY else planes
    P = oracle_pool(kind, (layers, heads, dim, blocks, page, planes))
    D = sentinel_destination(kind, (layers, heads, dim, blocks, page, planes), planes=dst_planes)
    P.fill_random(np.random.default_rng(len(name)))
    P.shuffle_free_list(rng)
    D.shuffle_free_list(rng)
    ranges, exits = [], []
    for i, n in enumerate(lengths):
        assert P.allocate(f"r{i}", n) and D.allocate(f"r{i}", n)
        ranges.append((min(i, n - 1), n))
        exits.append([rng.randrange(planes) for _ in range(n)])
        if mode == ho.MODE_DEDUP:
            for pos in range(n):
                P.finalize_token(f"r{i}", pos, exits[i][pos])
    tables = [[pool.plane_block_tables(f"r{i}") for i in range(len(lengths))] for pool in (P, D)]
    use = None if mode == ho.MODE_ALL_PLANES else exits
    side = torch.cuda.Stream()
    gp, gd = GpuPool(P), GpuPool(D)
    side.wait_stream(torch.cuda.current_stream())
    batch = k.HandoffBatch(*tables, ranges, block_size=page, exit_planes=use, src_blocks=blocks, dst_blocks=blocks)
    status = k.new_status()
    before = k.kernel_launches()
    k.kv_handoff(gp.view(), gd.view(), batch, mode=mode, status=status, stream=side)  # records sent on another stream
    side.synchronize()
    k.raise_for_status(status)
    assert k.kernel_launches() == before + 1
    for i, (s, e) in enumerate(ranges):
        ho.handoff_rows(P, D, tables[0][i], tables[1][i], s, e, mode=mode, exit_planes=exits[i])
    assert_pools_equal(gd, D)
    want = np.concatenate([ho.pack_rows(P, tables[0][i], s, e, mode=mode, exit_planes=exits[i]) for i, (s, e) in enumerate(ranges)])
    packed = torch.full((max(16, k.packed_bytes(gp.view(), batch.total_tokens, dst_planes)),), 0x5A, dtype=torch.uint8, device="cuda")
    workspace = k.dedup_workspace(batch, planes) if mode == ho.MODE_DEDUP else None
    before = k.kernel_launches()
    k.kv_pack(gp.view(), batch, packed, mode=mode, status=status, workspace=workspace)
    assert k.kernel_launches() == before + 1  # the wire plan is the host's: no plan kernels
    image = packed.cpu().numpy()
    assert np.array_equal(image[: want.size], want) and (image[want.size :] == 0x5A).all()
    if mode == ho.MODE_DEDUP:
        assert k.dedup_wire_tokens(workspace) == sum(exits[i][t] + 1 for i, (s, e) in enumerate(ranges) for t in range(s, e))
    for t in gd.tensors():
        t.view(torch.uint8).fill_(0x11)
    k.kv_scatter(packed, gd.view(), batch, mode=mode if mode == ho.MODE_DEDUP else 0, status=status, workspace=workspace)
    k.raise_for_status(status)
    for t in D.tensors(travelling_only=False):
        t.data[:] = 0x11
    for i, (s, e) in enumerate(ranges):
        ho.handoff_rows(P, D, tables[0][i], tables[1][i], s, e, mode=mode, exit_planes=exits[i])
    assert_pools_equal(gd, D)


@pytest.mark.parametrize("wide", ["source", "destination"])
def test_a_batch_with_more_planes_on_the_side_that_an_image_does_not_touch(wide):
    """A dedup image of three planes, packed or scattered with a batch that also holds tables of 70 planes for the other side."""
    from vllm_rlt_b200.kernels import kv_handoff as k

    page, planes, many, lengths = 4, 3, 70, [30, 9]
    P = oracle_pool("bf16", (2, 1, 16, 64, page, planes))
    D = sentinel_destination("bf16", (2, 1, 16, 64, page, planes))
    P.fill_random(np.random.default_rng(1))
    rng, exits, others = random.Random(1), [], []
    for i, n in enumerate(lengths):
        assert P.allocate(f"r{i}", n) and D.allocate(f"r{i}", n)
        exits.append([rng.randrange(planes) for _ in range(n)])
        others.append([[rng.randrange(64) for _ in range(-(-n // page))] for _ in range(many)])
        for pos in range(n):
            P.finalize_token(f"r{i}", pos, exits[i][pos])
    src, dst = ([pool.plane_block_tables(f"r{i}") for i in range(len(lengths))] for pool in (P, D))
    ranges = [(0, n) for n in lengths]
    gp, gd = GpuPool(P), GpuPool(D)
    pack = k.HandoffBatch(src, others if wide == "destination" else None, ranges, block_size=page, exit_planes=exits)
    scatter = k.HandoffBatch(others if wide == "source" else None, dst, ranges, block_size=page, exit_planes=exits)
    status = k.new_status()
    packed = torch.zeros(k.packed_bytes(gp.view(), pack.total_tokens, planes), dtype=torch.uint8, device="cuda")
    k.kv_pack(gp.view(), pack, packed, mode=k.MODE_DEDUP, status=status, workspace=k.dedup_workspace(pack, planes))
    want = np.concatenate([ho.pack_rows(P, t, s, e, mode=ho.MODE_DEDUP, exit_planes=x) for t, (s, e), x in zip(src, ranges, exits)])
    assert np.array_equal(packed.cpu().numpy()[: want.size], want)
    k.kv_scatter(packed, gd.view(), scatter, mode=k.MODE_DEDUP, status=status, workspace=k.dedup_workspace(scatter, planes))
    k.raise_for_status(status)
    for i, (s, e) in enumerate(ranges):
        ho.handoff_rows(P, D, src[i], dst[i], s, e, mode=ho.MODE_DEDUP, exit_planes=exits[i])
    assert_pools_equal(gd, D)


@pytest.mark.parametrize("layers", [255, 256, 300])  # 4,096 pairs a page: 32-bit division of (layer, pair) ends at 256 layers
def test_a_dedup_pack_of_many_layers_of_full_pages_on_many_planes(layers):
    from vllm_rlt_b200.kernels import kv_handoff as k

    planes = page = 64
    key, value = (torch.randint(-30000, 30000, (planes + 1, layers, page, 1, 1), dtype=torch.int16, device="cuda") for _ in range(2))
    blocks = torch.randperm(planes + 1)[:planes]
    exits = torch.randint(0, planes, (page,))
    exits[:60] = planes - 1
    view = k.PoolView.from_tensors(key.view(torch.bfloat16), value.view(torch.bfloat16), planes)
    batch = k.HandoffBatch([[[b] for b in blocks.tolist()]], None, [(0, page)], block_size=page, exit_planes=[exits.tolist()])
    want = torch.cat([t[b, :, (exits >= p).cuda()].reshape(-1) for p, b in enumerate(blocks.tolist()) for t in (key, value)])
    packed = torch.zeros(k.packed_bytes(view, page, planes), dtype=torch.uint8, device="cuda")
    status, workspace = k.new_status(), k.dedup_workspace(batch, planes)
    k.kv_pack(view, batch, packed, mode=k.MODE_DEDUP, status=status, workspace=workspace)
    k.raise_for_status(status)
    assert torch.equal(packed.view(torch.int16)[: want.numel()], want)
