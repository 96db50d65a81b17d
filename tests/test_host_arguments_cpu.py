"""Arguments that the compiled host side must not take for others: fractions, positions whose end does not fit 64 bits, ranges that
wrap around, ranges without tables."""

import struct

import numpy as np
import pytest
import torch

from tests.test_chunk_descriptors_cpu import descriptor, pulled
from tests.test_staging_cpu import st  # noqa: F401  (fixture)


def test_a_staged_write_starts_at_a_whole_position_inside_its_row(st):  # noqa: F811
    table = torch.zeros(3, 8, dtype=torch.int32)
    writer = st.StagedWriteTensor(table, 2, 4)
    for start in (2**63 - 1, 2**63 - 2, 8, -1):
        with pytest.raises(ValueError, match="outside the target row"):
            writer.stage_write(0, start, [1, 2])
    with pytest.raises(TypeError):
        writer.stage_write(0, 1.5, [1, 2])
    writer.stage_write(0, np.int64(6), [1, 2])
    writer.submit()
    assert table.tolist() == [[0] * 6 + [1, 2], [0] * 8, [0] * 8]


def test_a_chunk_range_is_given_in_whole_numbers():
    from vllm_rlt_b200.pd import transport

    tables = ((0, 1), (2, 3))
    for start, end, extra in ((0.5, 4, []), (0, 4.5, []), (0, 4, [(1, 2, 3.5)])):
        with pytest.raises(TypeError):
            transport.encode_chunk([(tables, tables, start, end)], extra)


@pytest.mark.parametrize("address, size", [((1 << 20) + 8, 2**63 - 16), (1 << 20, -1), (2**62, 2**62), ((1 << 21) + 1, 0)])
def test_a_range_that_wraps_around_is_not_inside_the_peers_memory(address, size):
    raw = bytearray(descriptor())
    struct.pack_into("<3q", raw, len(raw) - 24, address, 1 << 25, size)
    assert pulled(bytes(raw)) is None


def test_a_batch_without_tables_holds_no_records():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    batch = kh.HandoffBatch(None, None, [(0, 1 << 40)], block_size=16)
    assert batch.metadata_bytes == 0 and batch.total_tokens == 1 << 40



def test_two_threads_that_ask_for_a_views_struct_get_one_that_stays():
    from vllm_rlt_b200.kernels import kv_handoff as kh

    seen = []

    class View(kh.PoolView):
        def as_struct(self):
            struct = super().as_struct()
            if not seen:  # the other thread comes in between, and has used its address already
                seen.append(None)
                seen[0] = self._address()
            return struct

    view = View(kh.Region(4096, 8192, 384, 128, 32), None, 8, 4, 3, 2, 0)
    assert view._address() == seen[0] == view._address()

