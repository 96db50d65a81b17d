"""Wire images that end early: the rows that lie wholly before the end are packed and scattered, what lies behind it is neither written nor read, and the
status says so. Rows on 4-, 8- and 16-byte boundaries of the image, records that are parameters and records in device memory."""

import random

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PLANES = 3


def wire_rows(pools, tables, ranges, exits, mode, page):
    """(offset, bytes, tensor, plane, block, layer, token of the block, request, token) of every row, in wire order; and the image's size."""
    from vllm_rlt_b200.kernels import kv_handoff as kh

    rows, at = [], 0
    for r, (begin, end) in enumerate(ranges):
        for plane in range(1 if mode == kh.MODE_EXIT_ONLY else PLANES):
            for k in range(begin // page, -(-end // page)):
                tokens = [t for t in range(max(begin, k * page), min(end, (k + 1) * page)) if mode != kh.MODE_DEDUP or exits[r][t] >= plane]
                for i, pool in enumerate(pools):
                    size = pool.shape[3] * pool[0, 0, 0, 0].nbytes
                    for layer in range(pool.shape[1]):
                        for t in tokens:
                            source = exits[r][t] if mode == kh.MODE_EXIT_ONLY else plane
                            rows.append((at, size, i, plane, tables[r][source][k], layer, t % page, r, t))
                            at += size
    return rows, at


@pytest.mark.parametrize("heads, dim", [(3, 32), (2, 64), (4, 32)])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("page, layers, lengths", [(16, 5, [1, 16, 37, 70]), (1, 2, [430, 390])])
def test_rows_before_the_end(heads, dim, mode, page, layers, lengths):
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.kernels import kv_handoff as kh

    rng = random.Random(heads * dim + mode)
    gen = torch.Generator(device="cuda").manual_seed(mode)
    to = 1 if mode == kh.MODE_EXIT_ONLY else PLANES
    pages = [-(-n // page) for n in lengths]
    P = KVPool(layers, heads, dim, sum(pages) * PLANES, page, PLANES, kv_cache_dtype="fp8_e4m3")
    D = KVPool(layers, heads, dim, sum(pages) * to, page, to, kv_cache_dtype="fp8_e4m3")
    tensors = lambda p: [p.key_cache, p.value_cache, p.key_scale, p.value_scale]  # noqa: E731
    for t in tensors(P):
        t.view(torch.uint8).random_(0, 256, generator=gen)

    def deal(k):
        ids = rng.sample(range(sum(pages) * k), sum(pages) * k)
        return [[[ids.pop() for _ in range(n)] for _ in range(k)] for n in pages]

    src, dst = deal(PLANES), deal(to)
    ranges = [(min(i, n - 1), n) for i, n in enumerate(lengths)]
    exits = [[rng.randrange(PLANES) for _ in range(n)] for n in lengths]
    host = [t.view(torch.uint8).cpu().numpy().reshape(*t.shape[:4], -1) for t in tensors(P)]
    rows, whole = wire_rows(host, src, ranges, exits, mode, page)
    image = np.concatenate([host[i][block, layer, t].reshape(-1) for _, _, i, _, block, layer, t, _, _ in rows])
    assert image.size == whole

    def batch():
        return kh.HandoffBatch(src, dst, ranges, block_size=page, exit_planes=None if mode == kh.MODE_ALL_PLANES else exits)

    workspace = kh.dedup_workspace(batch(), PLANES) if mode == kh.MODE_DEDUP else None
    for short in (whole - whole // 3 & ~15, whole - 16 & ~15, 16):
        packed = torch.full((whole + 64,), 0x5A, dtype=torch.uint8, device="cuda")
        status = kh.new_status()
        b = batch()
        kh.kv_pack(kh.PoolView.from_cache(P), b, packed[:short], mode=mode, status=status, workspace=workspace)
        assert status[0] == 1  # a range that the image does not hold
        last = max((at + size for at, size, *_ in rows if at + size <= short), default=0)
        got = packed.cpu().numpy()
        assert np.array_equal(got[:last], image[:last]) and (got[last:] == 0x5A).all()
        assert bool(b._staged) == (page == 1)

        for t in tensors(D):
            t.view(torch.uint8).fill_(0xA5)
        want = [np.full((*t.shape[:4], t.element_size() * (t.shape[4] if t.dim() == 5 else 1)), 0xA5, np.uint8) for t in tensors(D)]
        for at, size, i, plane, block, layer, t, r, token in rows:
            if at + size > short:
                continue
            row = host[i][block, layer, t]
            for deeper in range(plane, PLANES) if mode == kh.MODE_DEDUP and plane == exits[r][token] else [plane]:
                want[i][dst[r][deeper][token // page], layer, t] = row
        status = kh.new_status()
        full = torch.from_numpy(np.concatenate([image, np.full(64, 0x33, np.uint8)])).cuda()
        kh.kv_scatter(full[:short], kh.PoolView.from_cache(D), batch(), mode=mode if mode == kh.MODE_DEDUP else kh.MODE_ALL_PLANES, status=status,
                      workspace=workspace)
        assert status[0] == 1
        for got, w in zip(tensors(D), want):
            assert np.array_equal(got.view(torch.uint8).cpu().numpy().reshape(w.shape), w)
