"""Dedup packs at every cut of their pages into shares: several shares a layer, several layers a share, launches too small for either, pages that
contribute far more or less than the others and none at all. The image is the one that torch indexing puts together."""

import random

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (layers, heads, dim, page, planes, element type), lengths, how deep the requests' tokens go
CASES = {
    "two shares a layer": ((24, 16, 128, 16, 4, "bf16"), [900, 600], "deep"),
    "four, and eight of a smaller launch": ((24, 16, 128, 16, 16, "bf16"), [200], "uniform"),
    "several layers": ((30, 3, 64, 16, 7, "bf16"), [500] * 9, "uniform"),
    "layers that do not divide": ((7, 1, 48, 64, 5, "bf16"), [300, 64, 1], "uniform"),
    "one layer each": ((24, 16, 128, 16, 4, "bf16"), [1200], "shallow"),
    "a few tokens": ((24, 16, 128, 16, 4, "bf16"), [5, 1, 17], "uniform"),
    "uneven": ((8, 16, 128, 16, 32, "bf16"), [160] * 12, "one deep"),
    "uneven, and none": ((5, 2, 64, 64, 9, "bf16"), [64, 64, 130, 1], "one without"),
    "codes and scales": ((24, 6, 64, 16, 5, "fp8"), [333, 80], "uniform"),
    "codes and scales at odd places": ((24, 5, 64, 16, 5, "fp8"), [333, 80], "uniform"),
    "64 planes": ((3, 2, 64, 8, 64, "bf16"), [40, 8], "deep"),
}


def exits_of(kind, rng, r, n, planes):
    if kind == "uniform":
        return [rng.randrange(planes) for _ in range(n)]
    if kind == "one without":
        return [-1] * n if r == 1 else [rng.choice([-1, 0, planes - 1]) for _ in range(n)]
    return [planes - 1 if kind == "deep" or (kind == "one deep" and r == 3) else 0] * n


@pytest.mark.parametrize("name", CASES)
def test_images_are_whole_at_every_cut(name):
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.kernels import kv_handoff as kh

    (layers, heads, dim, page, planes, kind), lengths, deep = CASES[name]
    rng = random.Random(name)
    gen = torch.Generator(device="cuda").manual_seed(len(name))
    pages = [-(-n // page) for n in lengths]
    blocks = sum(pages) * planes + 3
    pool = KVPool(layers, heads, dim, blocks, page, planes, kv_cache_dtype="fp8_e4m3" if kind == "fp8" else "auto")
    tensors = [pool.key_cache, pool.value_cache] + ([pool.key_scale, pool.value_scale] if kind == "fp8" else [])
    for t in tensors:
        t.view(torch.uint8).random_(0, 256, generator=gen)
    ids = rng.sample(range(blocks), blocks)
    tables = [[[ids.pop() for _ in range(k)] for _ in range(planes)] for k in pages]
    ranges = [(min(r, n - 1), n) for r, n in enumerate(lengths)]
    exits = [exits_of(deep, rng, r, n, planes) for r, n in enumerate(lengths)]

    parts = []
    for table, (begin, end), exit in zip(tables, ranges, exits):
        of = np.array(exit)
        for plane in range(planes):
            for k in range(begin // page, -(-end // page)):
                lo, hi = max(begin, k * page), min(end, (k + 1) * page)
                at = torch.from_numpy(np.flatnonzero(of[lo:hi] >= plane) + lo - k * page).cuda()
                parts += [t[table[plane][k]][:, at].contiguous().view(torch.uint8).reshape(-1) for t in tensors if len(at)]
    want = torch.cat(parts)

    view = kh.PoolView.from_cache(pool)
    batch = kh.HandoffBatch(tables, tables, ranges, block_size=page, exit_planes=exits)
    packed = torch.full((want.numel() + 64,), 0x5A, dtype=torch.uint8, device="cuda")
    status = kh.new_status()
    kh.kv_pack(view, batch, packed, mode=kh.MODE_DEDUP, status=status, workspace=kh.dedup_workspace(batch, planes))
    assert torch.equal(packed[: want.numel()], want) and bool((packed[want.numel() :] == 0x5A).all())
    if deep == "one without":
        assert status[0] == 3  # a token whose exit plane is none
    else:
        kh.raise_for_status(status)
