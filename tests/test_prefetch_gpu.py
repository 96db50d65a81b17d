"""Launches that move 32 MB and more ask for their source ahead of time, from their parameters alone: the bytes they leave behind, what they report
and what they leave alone are those of torch indexing, whatever the alignment, the pages that are partly in range and the ids that are no block's."""

import random

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (layers, heads, dim, page, element type): rows of 4 KiB, of 480 and of 48 bytes (16-byte accesses), of 20 (4-byte, which do not ask), FP8 with scales
SHAPES = {"4k": (24, 16, 128, 16, "bf16"), "480": (31, 5, 48, 64, "bf16"), "48": (48, 1, 24, 32, "bf16"), "20": (48, 1, 10, 64, "bf16"),
          "one token": (48, 16, 128, 1, "bf16"), "fp8": (48, 16, 128, 16, "fp8"), "fp8 odd": (48, 7, 48, 16, "fp8")}
PLANES = 4


def pool(shape, blocks, planes, fill, generator):
    from vllm_rlt_b200.core.kv_pool import KVPool

    layers, heads, dim, page, kind = shape
    p = KVPool(layers, heads, dim, blocks, page, planes, kv_cache_dtype="fp8_e4m3" if kind == "fp8" else "auto")
    for t in tensors(p):
        raw = t.view(torch.uint8)
        raw.random_(0, 256, generator=generator) if fill is None else raw.fill_(fill)
    return p


def tensors(p):
    return [p.key_cache, p.value_cache] + ([p.key_scale, p.value_scale] if p.key_scale is not None else [])


def equal(p, want):
    return all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(tensors(p), want))


@pytest.mark.parametrize("mode", ["all", "exit"])
@pytest.mark.parametrize("name", SHAPES)
def test_handoffs_pack_and_scatter(name, mode):
    from vllm_rlt_b200.kernels import kv_handoff as kh

    shape = SHAPES[name]
    layers, _, _, page, _ = shape
    rng = random.Random(name + mode)
    gen = torch.Generator(device="cuda").manual_seed(len(name))
    planes = 1 if mode == "exit" else PLANES
    row = sum(t[0, 0, 0].numel() * t.element_size() for t in tensors(pool(shape, 1, 1, 0, gen)))
    tokens = (40 << 20) // (2 * layers * row * planes) + 2 * page
    words = 6 + PLANES + planes + (page if mode == "exit" else 0)
    tokens = min(tokens, 7000 // words * page)  # the records stay parameters
    lengths = [tokens // 2 + 1, max(1, tokens // 3), page]
    pages = sum(-(-n // page) for n in lengths)
    src, dst = pool(shape, pages * PLANES + 3, PLANES, None, gen), pool(shape, pages * planes + 2, planes, 0xA5, gen)
    ids_s, ids_d = rng.sample(range(pages * PLANES + 3), pages * PLANES), rng.sample(range(pages * planes + 2), pages * planes)
    take = lambda ids, n, k: [[ids.pop() for _ in range(-(-n // page))] for _ in range(k)]  # noqa: E731
    st, dt = [take(ids_s, n, PLANES) for n in lengths], [take(ids_d, n, planes) for n in lengths]
    ranges = [(rng.randrange(min(n, page)), n) for n in lengths]
    exits = [[rng.randrange(PLANES) for _ in range(n)] for n in lengths] if mode == "exit" else None
    modes = kh.MODE_EXIT_ONLY if mode == "exit" else kh.MODE_ALL_PLANES
    sv, dv = kh.PoolView.from_cache(src), kh.PoolView.from_cache(dst)
    batch = kh.HandoffBatch(st, dt, ranges, block_size=page, exit_planes=exits)
    assert not batch._staged
    status = kh.new_status()

    def expect(skip=lambda r, plane, t: False):
        want = [torch.full_like(t.view(torch.uint8), 0xA5).view(t.dtype) for t in tensors(dst)]
        for r, (b, e) in enumerate(ranges):
            for plane in range(planes):
                at = torch.tensor([t for t in range(b, e) if not skip(r, plane, t)], device="cuda")
                from_plane = torch.tensor(exits[r], device="cuda")[at] if exits else torch.full_like(at, plane)
                sb = torch.tensor(st[r], device="cuda")[from_plane, at // page]
                db = torch.tensor(dt[r], device="cuda")[plane, at // page]
                for w, s in zip(want, tensors(src)):
                    w.view(torch.uint8)[db, :, at % page] = s.view(torch.uint8)[sb.clamp(max=src.num_blocks - 1), :, at % page]
        return want

    want = expect()
    for _ in range(3):  # one behind the other: the later ones ask while the one ahead still writes
        kh.kv_handoff(sv, dv, batch, mode=modes, status=status)
    kh.raise_for_status(status)
    assert equal(dst, want)
    packed = torch.zeros(kh.packed_bytes(sv, batch.total_tokens, planes), dtype=torch.uint8, device="cuda")
    kh.kv_pack(sv, batch, packed, mode=modes, status=status)
    for t in tensors(dst):
        t.view(torch.uint8).fill_(0xA5)
    kh.kv_scatter(packed, dv, batch, mode=kh.MODE_ALL_PLANES, status=status)
    kh.raise_for_status(status)
    assert equal(dst, want)

    # an id that is no block's: its rows stay out, the others arrive
    for t in tensors(dst):
        t.view(torch.uint8).fill_(0xA5)
    bad = (len(st[0][1]) // 2)
    st[0][1][bad] = src.num_blocks + 7
    if exits:
        exits[1][ranges[1][1] - 1] = 9
    with_bad = kh.HandoffBatch(st, dt, ranges, block_size=page, exit_planes=exits)
    kh.kv_handoff(sv, dv, with_bad, mode=modes, status=status)
    assert status[0] != 0
    if exits:
        last = ranges[1][1] - 1
        exits[1][last] = 0
        want = expect(lambda r, plane, t: (r == 0 and t // page == bad and exits[0][t] == 1) or (r == 1 and t == last))
    else:
        want = expect(lambda r, plane, t: r == 0 and plane == 1 and t // page == bad)
    assert equal(dst, want)


@pytest.mark.parametrize("shift", [0, 1, 4, 16, 31])
@pytest.mark.parametrize("odd", [0, 1, 15, 16384])
def test_byte_ranges(shift, odd):
    from vllm_rlt_b200 import _lib
    from vllm_rlt_b200.kernels import kv_handoff as kh

    n = (20 << 20) + odd
    src = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda")
    dst = torch.zeros(n + 64, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        kh.kv_push(src.data_ptr() + shift, dst.data_ptr() + 32, n)
    assert torch.equal(dst[32 : 32 + n], src[shift : shift + n]) and int(dst[:32].sum()) == 0 and int(dst[32 + n :].sum()) == 0
    dst.zero_()
    cuts = [0, 7, 40, 5 << 20, (5 << 20) + 16384, n]
    triples = np.array([(src.data_ptr() + shift + a, dst.data_ptr() + 32 + a, b - a) for a, b in zip(cuts, cuts[1:])], np.int64)
    _lib.check(_lib.load_host().copy_segments(triples.tobytes(), 0, None), "copy")
    assert torch.equal(dst[32 : 32 + n], src[shift : shift + n]) and int(dst[:32].sum()) == 0 and int(dst[32 + n :].sum()) == 0


@pytest.mark.parametrize("source, target, count", [(torch.float32, torch.bfloat16, 6_000_001), (torch.int64, torch.int32, 4_000_003),
                                                   (torch.bfloat16, torch.float32, 6_000_007), (torch.int32, torch.int32, 4_200_001)])
@pytest.mark.parametrize("skip", [0, 1, 3, 8])
def test_typed_copies(source, target, count, skip):
    from vllm_rlt_b200.worker.tensors import copy_tensor

    a = torch.randint(-(1 << 15), 1 << 15, (count + skip,), device="cuda").to(source)[skip:]
    out = torch.zeros(count + skip + 5, dtype=target, device="cuda")
    for _ in range(2):
        copy_tensor(a, out[skip : skip + count])
    assert torch.equal(out[skip : skip + count], a.to(target)) and int(out[:skip].abs().sum()) == 0 and int(out[skip + count :].abs().sum()) == 0
