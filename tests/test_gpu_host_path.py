"""What the native host path (csrc/sb_torch.cpp) owes its callers besides the numbers: the interpreter lock, memory, refusals."""
import os
import subprocess
import sys
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


@pytest.mark.parametrize("token_major", [False, True])
def test_rows_behind_the_last_sequence_are_filled_in_deterministic_mode(token_major):
    """torch.use_deterministic_algorithms fills new memory with NaN; the rows of o that no kernel writes hold what was allocated."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    cu = torch.tensor([0, 100, 256], device="cuda")
    q = torch.randn(2, 300, 64, device="cuda", dtype=torch.bfloat16)
    if token_major:
        q = q.transpose(0, 1).contiguous().transpose(0, 1)
    torch.full((2, 300, 64), 7.0, device="cuda", dtype=torch.bfloat16)  # what the next allocation of this size would find
    before = torch.are_deterministic_algorithms_enabled()
    torch.use_deterministic_algorithms(True)
    try:
        for x in (q, q.clone().requires_grad_()):
            o, _ = sb_attn_varlen(x, x, x, cu, 256)
            assert torch.isnan(o[:, 256:]).all() and torch.isfinite(o[:, :256].float()).all()
    finally:
        torch.use_deterministic_algorithms(before)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_memory_kept_for_the_backward(dtype):
    """o, rem and the forward workspace, nothing else: not neg_log_acc, which no backward reads."""
    from stickbreaking_attention_b200 import ops, sb_attn_varlen
    H, T, D = 4, 2000, 64
    x = torch.randn(H, T, D, device="cuda", dtype=dtype, requires_grad=True)
    cu = torch.tensor([900, T], device="cuda")

    def requested():
        return torch.cuda.memory_stats()["requested_bytes.all.current"]

    sb_attn_varlen(x, x, x, cu, 1100, zero_start=False)
    before = requested()
    out = sb_attn_varlen(x, x, x, cu, 1100, zero_start=False)
    workspace, _ = ops.workspace_bytes(False, 2, H, T, 1100)
    assert requested() - before == workspace + sum(y.numel() * y.element_size() for y in out)


def test_threads_without_a_current_context_take_the_tensor_core_kernels():
    """A thread whose first CUDA call is the operator's (its memory comes from the allocator's cache) has no current context when its
    tensor maps are encoded: a fresh Python thread, and the autograd thread of a process's first backward.  With the tensor-core path
    asked for, a refused map is an error and not a quiet change of kernels."""
    code = """
import threading, torch
from stickbreaking_attention_b200 import sb_attn_varlen, set_path
set_path("tensor")
q = torch.randn(2, 300, 64, device="cuda", dtype=torch.bfloat16, requires_grad=True)
cu = torch.tensor([100, 300], device="cuda")
results = []
def forward():
    o, rem = sb_attn_varlen(q, q, q, cu, 200, zero_start=False)
    results.append(o)
forward()
torch.cuda.synchronize()
x = [torch.empty(1 << 16, device="cuda") for _ in range(8)]  # for the cache
del x
thread = threading.Thread(target=forward)
thread.start()
thread.join()
g, = torch.autograd.grad(results[1], q, torch.ones_like(results[1]))
assert torch.equal(results[0], results[1]) and torch.isfinite(g.float()).all()
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
