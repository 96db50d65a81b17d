"""What a user of this library has it do, as measurable cases: one pass each through the public entry points.

Every case names an operation (``op``), a KV shape and sizes. The shapes are those of ``vllm_rlt_b200.workloads``
(Ouro-1.4B / 2.6B, FP8, Huginn-3.5B) and, in ``draw``, small and odd ones like those of the tests. KV values are N(0,1)
in bf16 or non-NaN e4m3 bytes with U[0.01, 0.1] scales; block tables are shuffled; exit planes are per token. All
operations move or convert values without arithmetic, so outputs are compared byte for byte.
"""

from __future__ import annotations

import math
import random
from types import SimpleNamespace

import numpy as np
import torch

from vllm_rlt_b200 import workloads
from vllm_rlt_b200.core.kv_pool import KVPool
from vllm_rlt_b200.kernels import kv_handoff as kh
from vllm_rlt_b200.pd.config import PDConfig
from vllm_rlt_b200.pd.transport import B200Transport
from vllm_rlt_b200.worker.staging import StagedInputTensor, StagedWriteTensor
from vllm_rlt_b200.worker.tensors import TensorTransfer, copy_tensor

_MODES = {"all": kh.MODE_ALL_PLANES, "dedup": kh.MODE_DEDUP, "exit_only": kh.MODE_EXIT_ONLY}
_DTYPES = {"int32": torch.int32, "int64": torch.int64, "float16": torch.float16, "bfloat16": torch.bfloat16,
           "float32": torch.float32}
_HIDDEN = 2048      # hidden size of the Ouro shapes: what one hidden-state row holds
_MOST_BYTES = 8e9   # a drawn case moves no more than this; the largest listed one moves about 9e9


def _shape(s: workloads.KVShape) -> dict:
    return dict(layers=s.num_layers, heads=s.num_kv_heads, dim=s.head_dim, planes=s.planes, block=s.block_size, fp8=s.fp8)


_OURO_1P4B, _OURO_2P6B = _shape(workloads.OURO_1P4B), _shape(workloads.OURO_2P6B)
_OURO_2P6B_FP8, _HUGINN = _shape(workloads.OURO_2P6B_FP8), _shape(workloads.HUGINN_3P5B)


def listed():
    return [
        # Layer streaming: what is left of one plane of a short prompt after its last layer. One launch, tables on the host.
        dict(name="streamed layer", op="slice", **_OURO_1P4B, tokens=200, group=1),
        # After every decode step: the tokens that left the recurrence early fill the deeper planes, one row per request.
        dict(name="decode step finalize", op="finalize", **_OURO_1P4B, requests=64, rows=1, prefix=24),
        # Before every decode step: token ids, positions, block-table updates and hidden rows of the running requests.
        dict(name="step metadata", op="staging", requests=48, tokens=1, writes=6, width=256),
        # A long prompt batch's token ids, narrowed on the device.
        dict(name="token ids narrowed", op="convert", count=1_000_003, source="int64", target="int32", second="none", skip=0),
        # One prompt handed from a four-plane pool to a single-plane one, tables straight from the two pools' allocators.
        dict(name="one prompt exit-only", op="handoff", **_OURO_1P4B, mode="exit_only", requests=1, shortest=1000, longest=1000,
             prefix=0, tables="pool"),
        # The end of a batch of prefills: every prompt token's exit-plane rows are copied to the deeper planes.
        dict(name="prompt finalize", op="finalize", **_OURO_1P4B, requests=4, rows=999, prefix=0),
        # The deployment's transfer: the prefill worker offers a prompt, the decode worker pulls it, both poll.
        dict(name="prompt pulled", op="transport", **_OURO_1P4B, tokens=777, form="tables", direction="pull"),
        # The same handover driven by the reference's connector: explicit descriptor lists, pushed chunk by chunk.
        dict(name="descriptors pushed", op="transport", **_OURO_1P4B, tokens=1000, form="descriptors", direction="push"),
        # FP8 codes with their scales, every plane, ragged prompts that share a prefix already resident on the decode side.
        dict(name="fp8 batch all planes", op="handoff", **_OURO_2P6B_FP8, mode="all", requests=6, shortest=128, longest=1500,
             prefix=256, tables="array"),
        # The staged path: distinct rows packed into a wire image, scattered on the other side with the copies rebuilt.
        dict(name="dedup wire image", op="wire", **_OURO_1P4B, mode="dedup", requests=4, shortest=512, longest=2048, prefix=0,
             tables="array"),
        # A recurrent-depth model: 32 planes, geometric exits, each distinct row read once and stored to every plane it fills.
        dict(name="recurrent depth dedup", op="handoff", **_HUGINN, mode="dedup", requests=2, shortest=300, longest=800, prefix=0,
             tables="array"),
        # The benchmark's workload at a size of which several fit one GPU.
        dict(name="batch exit-only", op="handoff", **_OURO_1P4B, mode="exit_only", requests=10, shortest=512, longest=4096,
             prefix=0, tables="array"),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_shape(rng):
    """Mostly the benchmark's shapes; sometimes a small or odd geometry of the kind the tests use."""
    pick = rng.random()
    if pick < 0.35:
        shape = dict(_OURO_1P4B)
    elif pick < 0.5:
        shape = dict(_OURO_2P6B)
    elif pick < 0.65:
        shape = dict(_OURO_2P6B_FP8)
    elif pick < 0.75:
        shape = dict(_HUGINN)
    else:
        shape = dict(layers=rng.randint(2, 48), heads=rng.randint(1, 16), dim=rng.choice([32, 48, 64, 80, 96, 128]),
                     planes=rng.randint(2, 8), block=rng.choice([8, 16, 32, 64]), fp8=rng.random() < 0.4)
    if rng.random() < 0.15:
        shape["block"] = rng.choice([8, 16, 32, 64])
    return shape


def draw(rng):
    op = rng.choice(["slice", "finalize", "finalize", "staging", "convert", "handoff", "handoff", "handoff", "wire", "transport",
                     "transport"])
    if op == "staging":
        return dict(op=op, requests=_log(rng, 1, 256), tokens=rng.choice([1, 1, 2, 5]), writes=rng.randint(1, 24),
                    width=_log(rng, 16, 2048))
    if op == "convert":
        names = list(_DTYPES)
        return dict(op=op, count=_log(rng, 1000, 1 << 27), source=rng.choice(names), target=rng.choice(names),
                    second=rng.choice(["none", "none", rng.choice(names)]), skip=rng.choice([0, 0, 0, 1]))
    shape = _draw_shape(rng)
    per_token = _plane_bytes(shape) * shape["planes"]
    if op == "slice":
        return dict(op=op, **shape, tokens=min(_log(rng, 16, 4096), int(_MOST_BYTES / 4 / per_token)),
                    group=rng.randint(1, min(12, shape["layers"])))
    if op == "finalize":
        requests = _log(rng, 1, 256)
        rows = 1 if rng.random() < 0.5 else _log(rng, 16, 2048)
        requests = max(1, min(requests, int(_MOST_BYTES / 2 / per_token / -(-rows // shape["block"]) / shape["block"])))
        rows = min(rows, int(_MOST_BYTES / 2 / per_token))
        return dict(op=op, **shape, requests=requests, rows=rows, prefix=rng.randint(0, 40))
    if op == "transport":
        return dict(op=op, **shape, tokens=max(16, min(_log(rng, 16, 2048), int(1.6e9 / per_token))),
                    form=rng.choice(["tables", "tables", "descriptors"]), direction=rng.choice(["pull", "push"]))
    mode = rng.choice(["all", "dedup"]) if op == "wire" else rng.choice(["all", "dedup", "exit_only"])
    requests, longest = _log(rng, 1, 64), _log(rng, 32, 4096)
    longest = max(16, min(longest, int(_MOST_BYTES / (4 if op == "wire" else 2) / per_token / requests)))
    requests = max(1, min(requests, int(_MOST_BYTES / (4 if op == "wire" else 2) / per_token / longest)))
    return dict(op=op, **shape, mode=mode, requests=requests, shortest=max(1, longest // rng.choice([1, 2, 8])), longest=longest,
                prefix=rng.choice([0, 0, 0, 4 * shape["block"]]), tables=rng.choice(["pool", "array"]))


# ------------------------------------------------------------------------------------------------ sizes


def _plane_bytes(c) -> int:
    """K and V of one token on one plane over all layers, scales included."""
    return 2 * c["layers"] * c["heads"] * (c["dim"] * (1 if c["fp8"] else 2) + (4 if c["fp8"] else 0))


def _lengths(c) -> list[int]:
    """Prompt lengths of a batch: part of the case, the same for every seed."""
    rng = random.Random(f"{c['requests']} {c['shortest']} {c['longest']}")
    return [rng.randint(c["shortest"], c["longest"]) for _ in range(c["requests"])]


def _exit_odds(planes: int) -> np.ndarray:
    """Probability of each zero-based exit plane: uniform for a few planes, geometric(0.1) from the fourth on for many
    (``workloads.recurrent_depth_dedup``)."""
    if planes <= 8:
        return np.full(planes, 1.0 / planes)
    tail = 0.9 ** np.arange(planes)  # P(exit recurrence > k)
    odds = tail - np.append(tail[1:], 0.0)
    odds[3] += odds[:3].sum()
    odds[:3] = 0.0
    return odds


def _exits(gen: np.random.Generator, planes: int, n: int) -> np.ndarray:
    return gen.choice(planes, size=n, p=_exit_odds(planes)).astype(np.int32)


def work(case):
    c = SimpleNamespace(**case)
    if c.op == "staging":
        values = c.requests * c.tokens
        return {"bytes": 2 * (values * 16 + c.requests * c.writes * 4 + c.requests * _HIDDEN * 2), "flops": 0}
    if c.op == "convert":
        size = sum(_DTYPES[n].itemsize for n in (c.source, c.target, c.second) if n != "none")
        return {"bytes": size * c.count, "flops": 0}
    token = _plane_bytes(case)
    odds = _exit_odds(c.planes)
    carried = float((odds * np.arange(1, c.planes + 1)).sum())  # planes that hold a row of their own, per token
    if c.op == "slice":
        return {"bytes": 2 * c.tokens * token // c.layers * c.group, "flops": 0}
    if c.op == "finalize":
        copies = float((odds * (c.planes - 1 - np.arange(c.planes))).sum())
        return {"bytes": c.requests * c.rows * token * (1.0 - odds[-1] + copies), "flops": 0}
    if c.op == "transport":
        return {"bytes": 2 * (c.tokens * token * c.planes + _HIDDEN * 2), "flops": 0}
    tokens = sum(_lengths(case))
    full = tokens * token * (1 if c.mode == "exit_only" else c.planes)
    distinct = tokens * token * carried if c.mode == "dedup" else full
    return {"bytes": 3 * distinct + full if c.op == "wire" else distinct + full, "flops": 0}


def tolerance(case):
    return "exact"


# ------------------------------------------------------------------------------------------------ states


def _pool(c, blocks, planes, gen, shuffle) -> KVPool:
    """A pool on the current GPU with shuffled free blocks: random KV if ``gen`` is given, zeros otherwise."""
    pool = KVPool(c.layers, c.heads, c.dim, blocks, c.block, planes, kv_cache_dtype="fp8_e4m3" if c.fp8 else "auto")
    for t in (pool.key_cache, pool.value_cache):
        if gen is None:
            t.view(torch.uint8).zero_()
        elif c.fp8:  # any e4m3 byte but the two NaN encodings, 0x7f and 0xff
            t.view(torch.int64).random_(generator=gen).bitwise_and_(0x7EFEFEFEFEFEFEFE)
        else:
            t.normal_(generator=gen)
    for t in (pool.key_scale, pool.value_scale) if c.fp8 else ():
        t.zero_() if gen is None else t.uniform_(0.01, 0.1, generator=gen)
    shuffle.shuffle(pool._free_blocks)
    return pool


def _pages(c, lengths):
    return sum(-(-n // c.block) for n in lengths)


def _bytes_of(pool) -> dict:
    """A pool's tensors as whole numbers: KV rows travel as bytes, and bytes are what is compared."""
    kind = torch.uint8 if pool.key_cache.element_size() == 1 else torch.int16
    out = dict(key=pool.key_cache.view(kind), value=pool.value_cache.view(kind))
    if pool.key_scale is not None:
        out.update(key_scale=pool.key_scale.view(torch.int32), value_scale=pool.value_scale.view(torch.int32))
    return out


def _prepare_batch(c, case, rngs):
    """Source and destination pools with their requests' tables, for handoffs and for the wire path."""
    lengths = [c.prefix + n for n in _lengths(case)]
    planes = 1 if c.mode == "exit_only" else c.planes
    pages = _pages(c, lengths)
    src = _pool(c, pages * c.planes, c.planes, rngs.device, rngs.host)
    dst = _pool(c, pages * planes, planes, None, rngs.host)
    tables = []
    for pool in (src, dst):
        for i, n in enumerate(lengths):
            assert pool.allocate(f"r{i}", n)
        rows = [pool.plane_block_tables(f"r{i}") for i in range(len(lengths))]
        if c.tables == "array":
            rows = [[np.array(t, np.int32) for t in request] for request in rows]
        tables.append(rows)
    exits = None
    if c.mode != "all":
        exits = [_exits(rngs.numbers, c.planes, n) for n in lengths]
    return SimpleNamespace(src=src, dst=dst, sv=kh.PoolView.from_cache(src), dv=kh.PoolView.from_cache(dst), src_tables=tables[0],
                           dst_tables=tables[1], ranges=[(c.prefix, n) for n in lengths], exits=exits, mode=_MODES[c.mode],
                           block=c.block, status=kh.new_status(), tokens=sum(lengths) - c.prefix * len(lengths))


def _batch(s):
    return kh.HandoffBatch(s.src_tables, s.dst_tables, s.ranges, block_size=s.block, exit_planes=s.exits,
                           src_blocks=s.src.num_blocks, dst_blocks=s.dst.num_blocks)


def _prepare_wire(c, case, rngs):
    s = _prepare_batch(c, case, rngs)
    batch = _batch(s)
    s.packed = torch.zeros(kh.packed_bytes(s.sv, s.tokens, c.planes), dtype=torch.uint8, device="cuda")
    s.workspace = kh.dedup_workspace(batch, c.planes) if c.mode == "dedup" else None
    return s


def _prepare_slice(c, case, rngs):
    pages = _pages(c, [c.tokens])
    s = SimpleNamespace(src=_pool(c, pages * c.planes, c.planes, rngs.device, rngs.host),
                        dst=_pool(c, pages * c.planes, c.planes, None, rngs.host), status=kh.new_status())
    s.tables = []
    for pool in (s.src, s.dst):
        assert pool.allocate("r", c.tokens)
        s.tables.append(np.array([pool.plane_block_tables("r")], np.int32))
    s.sv, s.dv = kh.PoolView.from_cache(s.src), kh.PoolView.from_cache(s.dst)
    s.begin, s.end = np.zeros(1, np.int32), np.array([c.tokens], np.int32)
    s.where = dict(layer_begin=c.layers - c.group, layer_end=c.layers, plane_begin=c.planes - 1, plane_end=c.planes)
    return s


def _prepare_finalize(c, case, rngs):
    """``rows`` consecutive tokens of every request, behind ``prefix`` pages of a prompt that all of them share."""
    pages = -(-c.rows // c.block)
    pool = _pool(c, (pages * c.requests + c.prefix) * c.planes, c.planes, rngs.device, rngs.host)
    shared = ()
    if c.prefix:
        assert pool.allocate("prefix", c.prefix * c.block)
        shared = tuple(zip(*pool.plane_block_tables("prefix")))
    rows, tables = [], []
    for i in range(c.requests):
        assert pool.allocate(f"r{i}", (c.prefix + pages) * c.block, prefix=shared)
        tables.append(pool.plane_block_tables(f"r{i}"))
        first = c.prefix * c.block + rngs.host.randint(0, pages * c.block - c.rows)
        rows.append(np.stack([np.full(c.rows, i, np.int32), _exits(rngs.numbers, c.planes, c.rows),
                              np.arange(first, first + c.rows, dtype=np.int32)], 1))
    view = kh.PoolView.from_tensors(pool.key_cache, pool.value_cache, c.planes, pool.key_scale, pool.value_scale)
    return SimpleNamespace(pool=pool, view=view, tables=torch.tensor(tables, dtype=torch.int32, device="cuda"),
                           rows=torch.from_numpy(np.concatenate(rows)).cuda(), status=kh.new_status())


def _prepare_transport(c, case, rngs):
    """A prefill and a decode worker on one GPU. A prompt leaves in chunks of at most ``transfer_chunk_bytes``: as one
    grouped launch in the table form, as submissions of whole blocks and partial rows in the descriptor form."""
    config = PDConfig()
    pages = _pages(c, [c.tokens])
    s = SimpleNamespace(config=config, src=_pool(c, pages * c.planes, c.planes, rngs.device, rngs.host),
                        dst=_pool(c, pages * c.planes, c.planes, None, rngs.host), form=c.form, passes=0)
    s.hidden_p = torch.randn(8, _HIDDEN, device="cuda", generator=rngs.device).to(torch.bfloat16)
    s.hidden_d = torch.zeros_like(s.hidden_p)
    s.p = B200Transport("prefill-0", s.src, s.hidden_p, config, direction=c.direction)
    s.d = B200Transport("decode-0", s.dst, s.hidden_d, config, lane=9, direction=c.direction)
    s.p.connect(s.d.info)
    s.d.connect(s.p.info)
    for pool in (s.src, s.dst):
        assert pool.allocate("r", c.tokens)
    s.tables = (s.src.plane_block_tables("r"), s.dst.plane_block_tables("r"))
    s.tokens, row = c.tokens, s.p.info["hidden_bytes"]
    hidden = (s.p.info["hidden_ptr"] + row, s.d.info["hidden_ptr"] + 2 * row, row)
    token = _plane_bytes(case) * c.planes
    if c.form == "tables":
        most = max(1, config.transfer_chunk_bytes // token)
        sizes = [min(most, c.tokens - at) * token for at in range(0, c.tokens, most)]
        if sizes[-1] + row > config.transfer_chunk_bytes:
            sizes.append(0)
        sizes[-1] += row
        s.parts, s.size, s.extra = list(enumerate(sizes)), sum(sizes), [hidden]
        s.notes = len(sizes)
    else:
        ranges = []
        for here, there in zip(*s.tables):
            for page, (a, b) in enumerate(zip(here, there)):
                held = min(c.block, c.tokens - page * c.block)
                for x, y in zip(_bytes_of(s.src).values(), _bytes_of(s.dst).values()):
                    size = x.element_size()
                    block, layer, one = (size * n for n in x.stride()[:3])
                    src, dst = x.data_ptr() + a * block, y.data_ptr() + b * block
                    if held == c.block:
                        ranges.append((src, dst, block))
                    else:
                        ranges += [(src + k * layer, dst + k * layer, held * one) for k in range(c.layers)]
        ranges.append(hidden)
        s.chunks, local, remote, total = [], [], [], 0
        for src, dst, n in ranges:
            if local and (total + n > config.transfer_chunk_bytes or len(local) == config.max_transfer_descriptors):
                s.chunks.append((local, remote, total))
                local, remote, total = [], [], 0
            local.append((src, n, 0))
            remote.append((dst, n, 0))
            total += n
        s.chunks.append((local, remote, total))
        s.notes = len(s.chunks)
    return s


def _prepare_staging(c, case, rngs):
    n = c.requests
    s = SimpleNamespace(n=n, tokens=c.tokens)
    s.ids = [rngs.numbers.integers(0, 50000, c.tokens).tolist() for _ in range(n)]
    s.positions = [list(range(p, p + c.tokens)) for p in rngs.numbers.integers(0, 4000, n).tolist()]
    s.input_ids, s.input_positions = StagedInputTensor(torch.int64, "cuda:0"), StagedInputTensor(torch.int64, "cuda:0")
    s.block_table = torch.zeros(n, c.width, dtype=torch.int32, device="cuda:0")
    s.table_writer = StagedWriteTensor(s.block_table, 16, 64)
    writes = min(c.writes, c.width)
    s.updates = [(i, rngs.host.randint(0, c.width - writes), rngs.numbers.integers(0, 1 << 20, writes).tolist()) for i in range(n)]
    s.hidden = torch.randn(n, _HIDDEN, device="cuda:0", generator=rngs.device).to(torch.bfloat16)
    s.hidden_rows = torch.zeros_like(s.hidden)
    s.row_of = rngs.numbers.permutation(n).tolist()
    s.mover = TensorTransfer(n, torch.bfloat16, "cuda:0")
    return s


def _prepare_convert(c, case, rngs):
    """Token ids and positions as integers, activations as floats; a conversion to int32 gets values that fit."""
    n = c.count + c.skip
    kind = _DTYPES[c.source]
    if kind.is_floating_point:
        source = torch.randn(n, device="cuda", generator=rngs.device).mul_(100.0).to(kind)
    else:
        source = torch.randint(-(1 << 15), 1 << 15 if "float16" in (c.target, c.second) else 1 << 20, (n,), dtype=kind,
                               device="cuda", generator=rngs.device)
    outs = [torch.zeros(n, dtype=_DTYPES[x], device="cuda") if x != "none" else None for x in (c.target, c.second)]
    cut = lambda t: None if t is None else t[c.skip :]  # noqa: E731  (skip = 1: a view that starts between two vectors)
    return SimpleNamespace(source=cut(source), target=cut(outs[0]), second=cut(outs[1]))


_PREPARE = dict(handoff=_prepare_batch, wire=_prepare_wire, slice=_prepare_slice, finalize=_prepare_finalize,
                transport=_prepare_transport, staging=_prepare_staging, convert=_prepare_convert)


def prepare(case, seed):
    torch.cuda.set_device(0)
    rngs = SimpleNamespace(device=torch.Generator(device="cuda").manual_seed(seed), numbers=np.random.default_rng(seed),
                           host=random.Random(seed))
    c = SimpleNamespace(**case)
    return c.op, _PREPARE[c.op](c, case, rngs)


# ------------------------------------------------------------------------------------------------ passes


def _run_handoff(s):
    kh.kv_handoff(s.sv, s.dv, _batch(s), mode=s.mode, status=s.status)
    return _bytes_of(s.dst)


def _run_wire(s):
    batch = _batch(s)
    kh.kv_pack(s.sv, batch, s.packed, mode=s.mode, status=s.status, workspace=s.workspace)
    kh.kv_scatter(s.packed, s.dv, batch, mode=s.mode, status=s.status, workspace=s.workspace)
    return dict(_bytes_of(s.dst), packed=s.packed)


def _run_slice(s):
    kh.kv_handoff_host(s.sv, s.dv, *s.tables, s.begin, s.end, status=s.status, **s.where)
    return _bytes_of(s.dst)


def _run_finalize(s):
    kh.kv_finalize(s.view, s.tables, s.rows, status=s.status)
    return _bytes_of(s.pool)


def _run_transport(s):
    """Submit one prompt, then poll both workers until the receiver has reported it and the sender's tickets are done."""
    s.passes += 1
    tid, notes = f"request-{s.passes}", 0
    if s.form == "tables":
        s.p.submit_tables(tid, 0, "decode-0", [(*s.tables, 0, s.tokens)], s.size, extra=s.extra, parts=s.parts)
    else:
        for sequence, (local, remote, size) in enumerate(s.chunks):
            while not s.p.submit(tid, sequence, "decode-0", local, remote, size):
                s.p.poll()
                notes += len(s.d.poll()[1])
    while notes < s.notes or s.p.pending:
        notes += len(s.d.poll()[1])
        s.p.poll()
    return dict(_bytes_of(s.dst), hidden=s.hidden_d)


def _run_staging(s):
    s.input_ids.reset()
    s.input_positions.reset()
    for ids, positions in zip(s.ids, s.positions):
        s.input_ids.append(ids)
        s.input_positions.append(positions)
    ids, positions = s.input_ids.upload(), s.input_positions.upload()
    s.table_writer.reset()
    for row, start, blocks in s.updates:
        s.table_writer.stage_write(row, start, blocks)
    s.table_writer.submit()
    s.mover.reset()
    for i, row in enumerate(s.row_of):
        s.mover.append(s.hidden[i], s.hidden_rows[row])
    s.mover.submit()
    return dict(ids=ids, positions=positions, block_table=s.block_table, hidden=s.hidden_rows)


def _run_convert(s):
    copy_tensor(s.source, s.target, secondary=s.second)
    return [s.target] if s.second is None else [s.target, s.second]


_RUN = dict(handoff=_run_handoff, wire=_run_wire, slice=_run_slice, finalize=_run_finalize, transport=_run_transport,
            staging=_run_staging, convert=_run_convert)


def run(state):
    op, s = state
    return _RUN[op](s)
