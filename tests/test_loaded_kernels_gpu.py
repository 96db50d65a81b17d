"""A new worker's first chunk of any kind is queued behind what runs on the GPU: the host does not wait for a kernel to be loaded."""

import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

# A process of its own, because a kernel is loaded once: what the worker has not loaded is loaded by its first launch.
PROGRAM = """
import sys
import torch
from tests.test_transport_gpu import drain
from vllm_rlt_b200.core.kv_pool import KVPool
from vllm_rlt_b200.pd.config import PDConfig
from vllm_rlt_b200.pd.transport import B200Transport
from vllm_rlt_b200.kernels import kv_handoff as kh

mode, tokens, planes = map(int, sys.argv[1:])
P, D = (KVPool(3, 4, 32, 5 * planes, 16, planes, device="cuda:0") for _ in range(2))
for t in (P.key_cache, P.value_cache):
    t.view(torch.uint8).random_(0, 256)
hidden = torch.zeros(2, 64, dtype=torch.bfloat16, device="cuda")
p = B200Transport("p0", P, hidden, PDConfig(), direction="push")
d = B200Transport("d0", D, hidden.clone(), PDConfig(), lane=9, direction="push")
p.connect(d.info)
d.connect(p.info)
assert P.allocate("a", tokens) and D.allocate("a", tokens)
requests = [(P.plane_block_tables("a"), D.plane_block_tables("a")[: 1 if mode == kh.MODE_EXIT_ONLY else None], 0, tokens)]
exits = None if mode == kh.MODE_ALL_PLANES else [[t % planes for t in range(tokens)]]
torch.cuda._sleep(1000)
torch.cuda.synchronize()
torch.cuda._sleep(1_000_000_000)  # about half a second of the device's clock
ahead = torch.cuda.Event()
ahead.record()
assert p.submit_tables("a", 0, "d0", requests, 100, mode=mode, exit_planes=exits, after=ahead)
waited = ahead.query()
assert drain(p, d, 1) == [("p0", "a", 0)]
p.close()
d.close()
print("WAITED" if waited else "QUEUED")
"""


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("tokens, planes", [(60, 64), (20, 65)])  # more than 64 planes are another file's kernels
def test_first_chunks_are_queued(mode, tokens, planes):
    done = subprocess.run([sys.executable, "-c", PROGRAM, str(mode), str(tokens), str(planes)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert done.stdout.split()[-1] == "QUEUED"
