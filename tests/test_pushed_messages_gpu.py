"""A pushed chunk is two launches: the copy, and the message with the ranges that ride along. Ranges that are many or large get their own."""

import pytest
import torch

from tests.test_transport_gpu import drain, expected_destination, make_pool, tensors

pytestmark = pytest.mark.gpu


# sizes of the ranges: none, odd ones, one block's worth, the most that ride along, one more byte, one more range
@pytest.mark.parametrize("sizes, ride", [([], True), ([1], True), ([4096], True), ([8192, 0, 33, 5], True), ([1 << 15], True),
                                         ([(1 << 15) + 1], False), ([1 << 14, (1 << 14) + 1], False), ([7] * 4, True), ([7] * 5, False)])
@pytest.mark.parametrize("shift", [0, 1, 16])
def test_ranges_and_message_travel_behind_the_tables(sizes, ride, shift):
    from vllm_rlt_b200.kernels import kv_handoff as kh
    from vllm_rlt_b200.pd.config import PDConfig
    from vllm_rlt_b200.pd.transport import B200Transport

    P, D = make_pool("cuda:0", seed=1), make_pool("cuda:0", seed=2, fill=False)
    hidden_p = torch.randint(-128, 128, (2, 1 << 16), dtype=torch.int8, device="cuda").view(torch.bfloat16)
    hidden_d = torch.zeros_like(hidden_p)
    p = B200Transport("p0", P, hidden_p, PDConfig(), direction="push")
    d = B200Transport("d0", D, hidden_d, PDConfig(), lane=9, direction="push")
    p.connect(d.info)
    d.connect(p.info)
    assert P.allocate("a", 70) and D.reserve_transfer("a", 70) is not None
    want = expected_destination(P, D, [("a", 3, 70)])
    src, dst = (t.view(torch.int8).reshape(-1) for t in (hidden_p, hidden_d))
    extra, expect, at = [], torch.zeros_like(dst), 0
    for n in sizes:
        extra.append((src.data_ptr() + at + shift, dst.data_ptr() + at, n))
        expect[at : at + n] = src[at + shift : at + shift + n]
        at += -(-n // 32) * 32 + 32
    requests = [(P.plane_block_tables("a"), D.plane_block_tables("a"), 3, 70)]
    for turn in range(3):
        before = kh.kernel_launches()
        assert p.submit_tables("a", turn, "d0", requests, 100, extra=extra)
        assert kh.kernel_launches() - before == (2 if ride else 2 + len(sizes))
        assert drain(p, d, 1) == [("p0", "a", turn)]
        torch.cuda.synchronize()
        for got, exp in zip(tensors(D), want):
            assert torch.equal(got.view(torch.uint8), exp.view(torch.uint8))
            got.view(torch.uint8).fill_(0xA5)
        assert torch.equal(dst, expect)
        dst.zero_()
    p.close()
    d.close()
