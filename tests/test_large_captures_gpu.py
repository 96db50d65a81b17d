"""CUDA graphs over launches that move 32 MB and more, whose host side looks addresses up; and a worker that is made while another thread captures."""

import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 20 << 20


def launches():
    """name -> (source, target, launch on the current stream)."""
    from vllm_rlt_b200 import _lib
    from vllm_rlt_b200.kernels import kv_handoff as kh
    from vllm_rlt_b200.worker.tensors import copy_tensor

    def push(a, b):
        kh.kv_push(a.data_ptr(), b.data_ptr(), N)

    def ranges(a, b):
        cuts = [0, 5, 4096, N // 2, N]
        triples = np.array([(a.data_ptr() + x, b.data_ptr() + x, y - x) for x, y in zip(cuts, cuts[1:])], np.int64)
        stream = torch.cuda.current_stream().cuda_stream
        _lib.check(_lib.load_host().copy_segments(triples.tobytes(), 0, stream), "copy")

    def flat(a, b):
        copy_tensor(a.view(torch.int32), b.view(torch.int32))

    def handoff(a, b):
        pages = 20
        views = []
        for t in (a, b):
            k, v = (x.view(torch.bfloat16).view(pages, 4, 16, 16, 256) for x in t.chunk(2))
            views.append(kh.PoolView.from_tensors(k, v, 1, None, None))
        table = [[np.arange(pages, dtype=np.int32)]]
        kh.kv_handoff(*views, kh.HandoffBatch(table, table, [(0, pages * 16)], block_size=16))

    return dict(push=push, ranges=ranges, flat=flat, handoff=handoff)


@pytest.mark.parametrize("name", ["push", "ranges", "flat", "handoff"])
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_large_launches_in_a_graph(name, mode):
    launch = launches()[name]
    a, b, c = (torch.zeros(N, dtype=torch.uint8, device="cuda") for _ in range(3))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode=mode):
        launch(a, b)
        launch(b, c)
    for _ in range(3):
        a.random_(0, 256)
        graph.replay()
        assert torch.equal(a, c)


@pytest.mark.parametrize("planes", [2, 65])
def test_a_worker_made_while_another_thread_captures(planes):
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.pd.config import PDConfig
    from vllm_rlt_b200.pd.transport import B200Transport

    pool = KVPool(3, 4, 32, 8 * planes, 16, planes, device="cuda:0")
    hidden = torch.zeros(2, 64, dtype=torch.bfloat16, device="cuda")
    x = torch.zeros(1000, device="cuda")
    torch.cuda.synchronize()
    capturing, made, failed = threading.Event(), threading.Event(), []

    def make():
        capturing.wait(60)
        try:
            B200Transport("p0", pool, hidden, PDConfig(), direction="push").close()
        except Exception as e:  # noqa: BLE001  (whatever it is, the test says so)
            failed.append(e)
        made.set()

    thread = threading.Thread(target=make)
    thread.start()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.add_(1)
        capturing.set()
        assert made.wait(60)
        x.add_(1)
    thread.join()
    assert not failed
    graph.replay()
    assert float(x.sum()) == 2000
