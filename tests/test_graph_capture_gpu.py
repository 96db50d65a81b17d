"""CUDA graphs over batches whose tables the host holds: built before the capture or within it, travelling as kernel parameters or
through device memory. A replay moves what the pools hold then, however often the library has used its staging since."""

import random

import numpy as np
import pytest
import torch

from oracle import handoff_oracle as ho
from tests.conftest import oracle_pool
from tests.gpu_support import GpuPool

pytestmark = pytest.mark.gpu


def single_plane(pages):
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.kernels import kv_handoff as kh

    pools = [KVPool(1, 1, 16, pages + 1, 4, 1, device="cuda") for _ in range(3)]
    tables = [np.random.default_rng(i).permutation(pages).astype(np.int32).reshape(1, 1, pages) for i in range(3)]
    return pools, [kh.PoolView.from_cache(p) for p in pools], tables


def moved(pools, tables, a, b):
    x, y = (torch.from_numpy(t.reshape(-1)).cuda().long() for t in (tables[a], tables[b]))
    return torch.equal(pools[a].key_cache[x], pools[b].key_cache[y]) and torch.equal(pools[a].value_cache[x], pools[b].value_cache[y])


@pytest.mark.parametrize("variant", [0, 5])  # the record kernels, the table-driven ones
@pytest.mark.parametrize("within", [False, True])
@pytest.mark.parametrize("pages", [20, 1000])  # kernel parameters, device memory
def test_a_captured_handoff_replays_and_the_batch_still_serves_other_launches(pages, within, variant):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    pools, views, tables = single_plane(pages)
    status = kh.new_status()

    def build(a, b):
        return kh.HandoffBatch(tables[a], tables[b], [(0, 4 * pages)], block_size=4)

    def launch(first, second):
        kh.kv_handoff(views[0], views[1], first, status=status, variant=variant)
        kh.kv_handoff(views[1], views[2], second, status=status, variant=variant)

    batches = [] if within else [build(0, 1), build(1, 2)]
    if variant and not within:
        launch(*batches)  # the arrays of this form are sent at the first use
    graphs = [torch.cuda.CUDAGraph() for _ in range(2)]
    for graph in graphs:  # the second capture cannot count on what the first one sent
        with torch.cuda.graph(graph):
            if not batches:
                batches = [build(0, 1), build(1, 2)]
            launch(*batches)
    other = [kh.HandoffBatch(tables[2], tables[0], [(0, 4 * pages)], block_size=4) for _ in range(80)]
    for batch in other if variant else ():
        batch.as_struct()
    torch.cuda.synchronize()
    for replay in (graphs[0].replay, graphs[1].replay, graphs[0].replay, lambda: launch(*batches), graphs[1].replay):
        pools[0].key_cache.normal_()
        pools[0].value_cache.normal_()
        for p in pools[1:]:
            p.key_cache.zero_()
            p.value_cache.zero_()
        replay()
        torch.cuda.synchronize()
        assert moved(pools, tables, 0, 1) and moved(pools, tables, 1, 2)
    kh.raise_for_status(status)
    del graphs  # their staging is used by the next capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        again = [build(0, 1), build(1, 2)]
        launch(*again)
    for p in pools[1:]:
        p.key_cache.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert moved(pools, tables, 0, 1) and moved(pools, tables, 1, 2)


@pytest.mark.parametrize("tokens", [600, 750])  # the layout of the image is sent in the capture, and with 600 the records too
def test_a_dedup_pack_whose_image_is_laid_out_in_the_capture(tokens):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    planes = 4
    P = oracle_pool("bf16", (1, 1, 16, planes * tokens + 3, 1, planes))
    P.fill_random(np.random.default_rng(tokens))
    P.shuffle_free_list(random.Random(tokens))
    assert P.allocate("r", tokens)
    exits = [random.Random(5).choices(range(planes), k=tokens)]
    tables = [P.plane_block_tables("r")]
    gp = GpuPool(P)
    batch = kh.HandoffBatch(tables, None, [(0, tokens)], block_size=1, exit_planes=exits)
    workspace, status = kh.dedup_workspace(batch, planes), kh.new_status()
    packed = torch.zeros(kh.packed_bytes(gp.view(), tokens, planes), dtype=torch.uint8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kh.kv_pack(gp.view(), batch, packed, mode=kh.MODE_DEDUP, status=status, workspace=workspace)
    want = ho.pack_rows(P, tables[0], 0, tokens, mode=ho.MODE_DEDUP, exit_planes=exits[0])
    others = [kh.HandoffBatch(tables, None, [(0, tokens)], block_size=1, exit_planes=[[0] * tokens]) for _ in range(80)]
    assert len(others) == 80
    for _ in range(2):
        packed.zero_()
        graph.replay()
        kh.raise_for_status(status)
        assert np.array_equal(packed.cpu().numpy()[: want.size], want)


def test_what_cannot_be_captured_is_refused_and_the_capture_goes_on():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    pages = 1000
    pools, views, tables = single_plane(pages)
    begin, end = np.zeros(1, np.int32), np.full(1, 4 * pages, np.int32)
    pools[0].key_cache.normal_()
    pools[0].value_cache.normal_()
    batch = kh.HandoffBatch(tables[0], tables[1], [(0, 4 * pages)], block_size=4)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(RuntimeError):  # its staging is the library's, for one launch
            kh.kv_handoff_host(views[0], views[1], tables[0], tables[1], begin, end)
        kh.kv_handoff(views[0], views[1], batch)
    graph.replay()
    torch.cuda.synchronize()
    assert moved(pools, tables, 0, 1)


def test_a_batch_dropped_while_its_stream_captures_leaves_the_capture_alone():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    pages = 1000
    pools, views, tables = single_plane(pages)
    own, other = torch.cuda.Stream(), torch.cuda.Stream()
    pools[0].key_cache.normal_()
    pools[0].value_cache.normal_()
    torch.cuda.synchronize()
    dropped = kh.HandoffBatch(tables[0], tables[1], [(0, 4 * pages)], block_size=4, stream=own)
    kept = kh.HandoffBatch(tables[1], tables[2], [(0, 4 * pages)], block_size=4, stream=own)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=own):
        kh.kv_handoff(views[0], views[1], dropped, stream=other)  # outside the capture
        del dropped
        kh.kv_handoff(views[1], views[2], kept, stream=own)
    torch.cuda.synchronize()
    assert moved(pools, tables, 0, 1) and not moved(pools, tables, 1, 2)
    graph.replay()
    torch.cuda.synchronize()
    assert moved(pools, tables, 1, 2)
