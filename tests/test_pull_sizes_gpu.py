"""A pulled chunk at the sizes where its records change places: kernel parameters, the library's staging slot, the general path;
and one that the compiled call must leave to the general path, which says what is wrong."""

import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direction", ["pull", "push"])
@pytest.mark.parametrize("tokens", [1, 700, 3100, 7000])
def test_chunks_of_few_and_many_pages_arrive_whole(tokens, direction):
    from vllm_rlt_b200.core.kv_pool import KVPool
    from vllm_rlt_b200.pd.config import PDConfig
    from vllm_rlt_b200.pd.transport import B200Transport

    pages = -(-tokens // 4)  # 10 words a page: 7,680 words of parameters hold 768 pages, a slot 1,638
    P, D = (KVPool(2, 1, 16, 2 * pages + 2, 4, 2, device="cuda:0") for _ in range(2))
    for t in (P.key_cache, P.value_cache):
        t.normal_()
    for t in (D.key_cache, D.value_cache):
        t.zero_()
    D._free_blocks.reverse()
    assert P.allocate("r", tokens) and D.allocate("r", tokens)
    hidden = torch.arange(32, dtype=torch.bfloat16, device="cuda:0").reshape(2, 16)
    landed = torch.zeros_like(hidden)
    p = B200Transport("p0", P, hidden, PDConfig(), direction=direction)
    d = B200Transport("d0", D, landed, PDConfig(), lane=9, direction=direction)
    p.connect(d.info)
    d.connect(p.info)
    tables = P.plane_block_tables("r"), D.plane_block_tables("r")
    start = min(5, tokens - 1)
    size = (tokens - start) * 2 * 2 * 2 * 32 + 32
    assert p.submit_tables("r", 0, "d0", [(*tables, start, tokens)], size,
                           extra=[(p.info["hidden_ptr"] + 32, d.info["hidden_ptr"], 32)])
    notes, deadline = [], time.monotonic() + 20
    while (p.pending or not notes) and time.monotonic() < deadline:
        notes += d.poll()[1]
        p.poll()
    assert notes == [("p0", "r", 0)] and p.bytes_sent == size and d.bytes_received == (size if direction == "pull" else 0)
    at = torch.arange(start, tokens, device="cuda:0")
    for plane in range(2):
        a, b = (torch.tensor(t[plane], device="cuda:0")[at // 4] for t in tables)
        for x, y in ((P.key_cache, D.key_cache), (P.value_cache, D.value_cache)):
            assert torch.equal(x[a, :, at % 4], y[b, :, at % 4])
            y[b, :, at % 4] = 0
    assert torch.equal(landed[0], hidden[1])
    assert not any(bool(t.any()) for t in (D.key_cache, D.value_cache))
    if direction == "pull":
        broken = (tables[0], tuple(tuple(10**6 for _ in t) for t in tables[1]))
        assert p.submit_tables("bad", 0, "d0", [(*broken, 0, tokens)], size)
        torch.cuda.synchronize()
        with pytest.raises(ValueError, match="physical block outside registered pool"):
            d.poll()
        p.pending.clear()
    d.close()
    p.close()
