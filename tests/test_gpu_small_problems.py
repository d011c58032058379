"""Small forwards build the table of work items inside the kernel; larger ones take it from a kernel of its own."""
import numpy as np
import pytest
import torch

from util import synth

pytestmark = pytest.mark.gpu

PACKS = {
    "one": [1],
    "ragged": [130, 0, 257, 64, 1, 0, 128],
    "most_sequences": [(37 * i) % 200 for i in range(32)],   # 32 sequences: the last count that builds its own table
    "too_many": [(37 * i) % 200 for i in range(33)],
    "one_long": [128 * 96 + 5],
}


def _run(q, k, v, do, dr, cu, m):
    from stickbreaking_attention_b200 import launch_count, sb_attn_varlen
    q, k, v = (x.clone().requires_grad_() for x in (q, k, v))
    before = launch_count()
    o, rem = sb_attn_varlen(q, k, v, cu, m, zero_start=False)
    torch.cuda.synchronize()
    launches = launch_count() - before
    return launches, (o.detach(), rem.detach()) + torch.autograd.grad([o, rem], [q, k, v], [do, dr])


@pytest.mark.parametrize("dtype,cu_dtype", [(torch.bfloat16, torch.int32), (torch.bfloat16, torch.int64), (torch.float32, torch.int32)])
@pytest.mark.parametrize("name", sorted(PACKS))
def test_own_tables_give_the_same_bits(name, dtype, cu_dtype):
    """The first head alone (own table) against the same head among so many that the table kernel runs; tokens behind the last
    sequence included."""
    lengths, pad, D = PACKS[name], 7, 64
    T = sum(lengths) + pad
    H = 296 // (T // 128 + len(lengths)) + 1  # one head more than the rule allows
    q, k, v, do, dr = (torch.from_numpy(x).to("cuda", dtype) for x in synth(H, T, D, 41))
    cu = torch.tensor(np.cumsum(lengths), dtype=cu_dtype, device="cuda")
    m = max(lengths)
    n_all, want = _run(q, k, v, do, dr, cu, m)
    n_one, got = _run(q[:1], k[:1], v[:1], do[:1], dr[:1], cu, m)
    assert n_all == 2 and n_one == (2 if name == "too_many" else 1)
    covered = T - pad
    assert torch.equal(got[0][:, :covered], want[0][:1, :covered])  # rows of o behind the last sequence are left alone
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a, b[:1])


@pytest.mark.parametrize("name", sorted(set(PACKS) - {"too_many"}) + ["most_items"])
def test_blocks_of_own_tables_take_items_in_turn(name):
    """As many heads as still build their own table, on the tensor-core kernels up to two (item, head) pairs per SM: blocks then take a
    second one without a counter.  The same bits as among one head more, where the table kernel and the counter do it.  Packs of up to
    256 items: the most that the table in shared memory holds."""
    lengths, pad, D, dtype = PACKS.get(name, [128 * 249 + 5] + [1] * 6), 7, 64, torch.bfloat16
    T = sum(lengths) + pad
    items = T // 128 + len(lengths)  # the bound that the rule goes by
    assert items <= 256
    H = 296 // items
    q, k, v, do, dr = (torch.from_numpy(x).to("cuda", dtype) for x in synth(H + 1, T, D, 42))
    cu = torch.tensor(np.cumsum(lengths), dtype=torch.int32, device="cuda")
    n_all, want = _run(q, k, v, do, dr, cu, max(lengths))
    n_own, got = _run(*(x[:H] for x in (q, k, v, do, dr)), cu, max(lengths))
    assert n_all == 2 and n_own == 1
    covered = T - pad
    assert torch.equal(got[0][:, :covered], want[0][:H, :covered])
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a, b[:H])


def test_own_tables_report_bad_sequence_ends():
    import stickbreaking_attention_b200 as sb
    q = torch.randn(1, 256, 64, device="cuda", dtype=torch.bfloat16)
    sb.check_status()
    for ends, m in ([200, 100], 256), ([100, 300], 256), ([100, 256], 120):
        with pytest.raises(ValueError):
            sb.sb_attn_varlen(q, q, q, torch.tensor(ends, device="cuda"), m, zero_start=False)
            sb.check_status()
    assert sb.check_status() == 0


@pytest.mark.parametrize("cu_dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1000])
def test_sequence_bounds_read_from_the_device(n, cu_dtype):
    """First entry and longest sequence, exact, at both sides of the kernel's 256 threads; strided ends as well."""
    from stickbreaking_attention_b200 import _lib
    ends = np.cumsum(np.random.default_rng(n).integers(0, 90, n))
    cu = torch.from_numpy(ends).to("cuda", cu_dtype)
    strided = torch.stack([cu, cu], 1)[:, 0]
    for leading in (False, True):
        gaps = np.diff(ends) if leading else np.diff(ends, prepend=0)
        want = (int(ends[0]), int(gaps.max()) if len(gaps) else 0)
        assert _lib.binding().seq_bounds(cu, leading, True) == want
        assert _lib.binding().seq_bounds(strided, leading, True) == want
        assert _lib.binding().seq_bounds(cu, leading, False)[0] == want[0]
