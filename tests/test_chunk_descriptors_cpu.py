"""Chunk descriptors come out of memory that another process writes: one that is cut short, or that announces more than it holds,
is left to the general path before anything is allocated or queued for it."""

import ctypes as C
import struct
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def pulled(raw):
    """What the compiled call makes of a descriptor for a pool of 2 planes, 8 blocks of 4 tokens. It must not come as far as a launch."""
    from vllm_rlt_b200 import _lib

    region = _lib.RltRegion(4096, 8192, 3 * 4 * 32, 4 * 32, 32)
    pool = _lib.RltPool(region, _lib.RltRegion(None, None, 0, 0, 0), 8, 4, 3, 2)
    at = C.addressof(pool)
    return _lib.load_host().pull_chunk(at, at, raw, [(1 << 20, 1 << 21, 1 << 30)], 0, 0)


def descriptor():
    from vllm_rlt_b200.pd import transport

    tables = ((0, 1, 2), (3, 4, 5))
    return transport.encode_chunk([(tables, tables, 1, 11)], [(1 << 20, 1 << 25, 64)])


def test_a_descriptor_cut_short_anywhere_queues_nothing():
    raw = descriptor()
    assert all(pulled(raw[:n]) is None for n in range(len(raw)))


def test_a_descriptor_that_announces_more_ranges_than_it_holds_costs_no_memory():
    announced = []
    for count in (2, 1 << 20, (1 << 32) - 1):
        raw = bytearray(descriptor())
        struct.pack_into("<I", raw, 4, count)
        announced.append(bytes(raw).hex())
    # at most 2 GiB beyond what the process has already: the announced ranges would take up to 103 GB
    code = (
        "import resource\n"
        "from tests.test_chunk_descriptors_cpu import pulled\n"
        "assert pulled(b'') is None\n"
        "held = int(open('/proc/self/statm').read().split()[0]) * resource.getpagesize()\n"
        "resource.setrlimit(resource.RLIMIT_AS, (held + (2 << 30),) * 2)\n"
        f"assert all(pulled(bytes.fromhex(raw)) is None for raw in {announced})\n"
    )
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert done.returncode == 0, done.stderr[-2000:]
