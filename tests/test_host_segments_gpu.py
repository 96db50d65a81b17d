"""Byte ranges whose list the host holds: every alignment, empty ranges, tile edges, and the list sizes at which it changes places."""

import random

import pytest
import torch

pytestmark = pytest.mark.gpu

TILE = 16 * 1024


@pytest.mark.parametrize("count", [1, 32, 33, 256, 257, 1024, 1025])
def test_ranges_from_the_host_are_copied_exactly(count):
    from vllm_rlt_b200 import _lib

    rng = random.Random(count)
    sizes = [rng.choice([0, 1, 31, 32, 33, 4096, TILE - 1, TILE, TILE + 1, 3 * TILE + 17]) for _ in range(count)]
    source = torch.randint(0, 256, (sum(sizes) + 96 * count + 64,), dtype=torch.uint8, device="cuda")
    target = torch.full_like(source, 0xA5)
    want = target.clone()
    local, remote, at = [], [], 0
    for n in sizes:
        shift = rng.choice([0, 0, 0, 1, 4, 16])  # of both sides, or of one
        a, b = at + shift, at + (shift if rng.random() < 0.7 else 0)
        local.append((source.data_ptr() + a, n, 0))
        remote.append((target.data_ptr() + b, n, 0))
        want[b : b + n] = source[a : a + n]
        at += (n + 16 + 63) // 64 * 64
    host = _lib.load_host()
    packed = host.pack_segments(local, remote, [(target.data_ptr(), target.data_ptr() + target.numel(), target.data_ptr())])
    assert len(packed) == 24 * count
    _lib.check(host.copy_segments(packed, 0, None), "copy")
    assert torch.equal(target, want)
    with pytest.raises(ValueError, match="outside the peer's registered memory"):
        host.pack_segments(local, [(0, n, 0) for _, n, _ in remote], [(64, 128, 0)])
    with pytest.raises(ValueError, match="geometry"):
        host.pack_segments(local, remote[1:], [])
