"""What the native host path (csrc/sb_torch.cpp) owes its callers besides the numbers: the interpreter lock, memory, refusals."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_seqlens", [None, 256])
def test_other_threads_run_while_a_call_waits(max_seqlens):
    """A call that has to read cu_seqlens waits for the stream; a second Python thread goes on meanwhile."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    q = torch.randn(2, 256, 64, device="cuda", dtype=torch.bfloat16)
    cu = torch.tensor([0, 100, 256], device="cuda")
    sb_attn_varlen(q, q, q, cu, max_seqlens)
    torch.cuda.synchronize()
    steps, stop = [0], threading.Event()

    def work():
        while not stop.wait(0.001):
            steps[0] += 1

    thread = threading.Thread(target=work)
    thread.start()
    try:
        while steps[0] == 0:
            time.sleep(0.001)
        torch.cuda._sleep(400_000_000)  # ~0.2 s
        before, start = steps[0], time.perf_counter()
        sb_attn_varlen(q, q, q, cu, max_seqlens)
        took, advanced = time.perf_counter() - start, steps[0] - before
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert took > 0.05  # the call did wait
    assert advanced >= 10, (took, advanced)
