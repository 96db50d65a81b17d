"""NumPy arrays of tables are read by their fields where they are plain int32, through the buffer protocol or a conversion otherwise: the same
values come out, and what is refused is the same."""

import array
import ctypes as C

import numpy as np
import pytest

ROWS = [[5, 1, 7], [2, 6, 3]]


def unaligned(values):
    raw = np.zeros(4 * len(values) + 1, np.uint8)
    out = raw[1:].view(np.int32)
    out[:] = values
    return out


class Sub(np.ndarray):
    pass


FORMS = {
    "list": lambda v: v,
    "int32": lambda v: np.array(v, np.int32),
    "read-only": lambda v: np.frombuffer(np.array(v, np.int32).tobytes(), np.int32),
    "strided": lambda v: np.repeat(np.array(v, np.int32), 3)[::3],
    "reversed": lambda v: np.array(v[::-1], np.int32)[::-1],
    "column": lambda v: np.array([v, v], np.int32, order="F")[0],
    "other byte order": lambda v: np.array(v, ">i4"),
    "int64": lambda v: np.array(v, np.int64),
    "uint32": lambda v: np.array(v, np.uint32),
    "int16": lambda v: np.array(v, np.int16),
    "subclass": lambda v: np.array(v, np.int32).view(Sub),
    "array.array": lambda v: array.array("i", v),
    "broadcast": lambda v: np.broadcast_to(np.int32(4), len(v)),
}


def records(tables, exits):
    """The padded arrays of the plan that the compiled host side makes of one request's tables."""
    from vllm_rlt_b200 import _lib

    host = _lib.load_host()
    plan = host.plan([tables], [tables], [(0, 6)], [exits], 2, 100, 100, 64)[0]
    size, offsets = host.plan_layout(plan)
    out = np.zeros(size, np.uint8)
    host.plan_arrays(plan, out)
    return out.tobytes(), offsets


@pytest.mark.parametrize("form", FORMS)
def test_tables_and_exit_planes_are_the_same_whatever_holds_them(form):
    rows = [[4, 4, 4]] * 2 if form == "broadcast" else ROWS
    exits = [4] * 6 if form == "broadcast" else [0, 1, 0, 1, 1, 0]
    assert records([FORMS[form](r) for r in rows], FORMS[form](exits)) == records(rows, exits)


@pytest.mark.parametrize("table", [np.zeros((3, 1), np.int32), np.zeros((), np.int32), np.zeros((3, 1), np.int64)])
def test_a_table_that_is_not_flat_is_refused(table):
    with pytest.raises(ValueError, match="flat sequence of block ids"):
        records([table, table], [0] * 6)


def test_a_table_between_two_words_is_refused():
    with pytest.raises(TypeError, match="must hold integers"):
        records([unaligned(r) for r in ROWS], [0] * 6)


def handed(*arrays):
    """What the compiled call makes of host arrays for pools of 2 planes, 8 blocks of 4 tokens that refuse every launch (no layers)."""
    from vllm_rlt_b200 import _lib

    region = _lib.RltRegion(4096, 8192, 3 * 4 * 32, 4 * 32, 32)
    pool = _lib.RltPool(region, _lib.RltRegion(None, None, 0, 0, 0), 8, 4, 0, 2)
    at = C.addressof(pool)
    return _lib.load_host().handoff_host(at, at, *arrays, 0, 0, 0, 0, None, 0)


def test_host_arrays_are_contiguous_int32_of_the_right_shape():
    tables, ends = np.zeros((2, 2, 3), np.int32), np.full(2, 3, np.int32)
    assert handed(tables, tables, ends * 0, ends) < 0  # looked over, and refused by the library for its pools
    assert handed(memoryview(tables), tables.view(Sub), array.array("i", [0, 0]), ends) < 0
    for bad in (np.zeros((2, 2, 3), ">i4"), np.zeros((2, 2, 3), np.int64), np.zeros((2, 2, 3), np.float32), np.zeros((2, 2, 6), np.int32)[:, :, ::2],
                np.zeros((3, 2, 2), np.int32).T, unaligned([0] * 12).reshape(2, 2, 3), [[[0] * 3] * 2] * 2):
        for side in ((bad, tables), (tables, bad)):
            with pytest.raises(ValueError, match="C-contiguous int32"):
                handed(*side, ends * 0, ends)
    for shapes in ((tables[0], tables, ends), (tables, tables[:1], ends), (tables, tables[:, :, :2].copy(), ends), (tables, tables, ends[:1])):
        with pytest.raises(ValueError, match=r"\[requests, planes, width\]|agree in requests and width"):
            handed(*shapes[:2], shapes[2] * 0, shapes[2])
