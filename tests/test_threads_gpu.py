"""Calls from threads that have made no other CUDA call."""

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_a_threads_first_call_may_be_a_product():
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    from toner_b200 import ops
    x = torch.randn(2, 96, 64, device="cuda").to(torch.bfloat16)
    outs = [torch.zeros(2, 64, 64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    failed = []

    def work(out):
        try:
            ops.syrk_upper(x, out, ops.EMA_FULL, 0.0, 1.0)
        except Exception as e:  # noqa: BLE001  (reported by the main thread)
            failed.append(e)

    work(outs[0])
    for out in outs[1:]:
        t = threading.Thread(target=work, args=(out,))
        t.start()
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    assert torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])
