"""Packs whose sequences have at most 128 tokens: the backward forms dq, dk and dv in one kernel."""
import math

import numpy as np
import pytest
import torch

from util import TOL_BF16, assert_close, oracle_varlen, rounded, synth, to_dev

pytestmark = pytest.mark.gpu

# the ends of slices of 16 rows, of 32-key quarters, of halves and of the tile
LENGTHS = [1, 128, 16, 15, 17, 31, 33, 63, 64, 65, 96, 97, 112, 113, 127]


@pytest.mark.parametrize("D,dtype,attend_current", [(128, torch.bfloat16, False), (128, torch.float16, True), (64, torch.bfloat16, True),
                                                    (32, torch.bfloat16, False)])
@pytest.mark.parametrize("fused", [False, True])
def test_sequences_of_one_tile(D, dtype, attend_current, fused):
    """Against the oracle, with NaN in the pad behind the last sequence (its gradients are zero)."""
    from stickbreaking_attention_b200 import launch_count, sb_attn_varlen
    H, T, pad = 3, sum(LENGTHS), 9
    ins = [rounded(x, dtype) for x in synth(H, T, D, seed=31)]
    q, k, v, do, dr = (torch.cat([to_dev(x, dtype), torch.full((H, pad) + x.shape[2:], float("nan"), dtype=dtype, device="cuda")], 1)
                       for x in ins)
    for x in (q, k, v):
        x.requires_grad_()
    cu = torch.tensor(np.cumsum(LENGTHS), dtype=torch.int32, device="cuda")
    it = 1 / math.sqrt(D)
    o, rem = sb_attn_varlen(q, k, v, cu, max(LENGTHS), zero_start=False, inv_temp=it, attend_current=attend_current, fuse_remainder=fused)
    before = launch_count()
    dq, dk, dv = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
    torch.cuda.synchronize()
    assert launch_count() - before == (2 if fused else 1)
    for g in (dq, dk, dv):
        assert torch.all(g[:, T:] == 0)
    qn, kn, vn, don, drn = ins
    if fused:  # out = o + rem v: drem receives do . v, dv receives rem do
        drn = drn + (don.astype(np.float64) * vn).sum(-1)
    want = list(oracle_varlen(qn, kn, vn, don, drn, LENGTHS, it, attend_current))
    if fused:
        want[0] = want[0] + want[1][..., None] * vn
        want[4] = want[4] + want[1][..., None] * don
    got = [x[:, :T].detach().double().cpu().numpy() for x in (o, rem, dq, dk, dv)]
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11  # what storing the exact result in the output type costs
    assert_close(("o", "rem", "dq", "dk", "dv"), got, want, TOL_BF16, f"one tile {D} {dtype} {fused}", out_half_ulp=half_ulp)


@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (64, torch.float16), (32, torch.bfloat16)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_rows_behind_a_sequence_see_no_key(D, dtype, bad):
    """The last key of every sequence is visible to no query: whatever its k holds, o, rem, dk and dv are the same bits.  (The rows of a
    tile between the end of the sequence and the next multiple of 16 lie behind that key and are part of the contractions.)"""
    from stickbreaking_attention_b200 import sb_attn_varlen
    lengths = [n for n in LENGTHS if n % 16]
    ends = np.cumsum(lengths)
    ins = [to_dev(rounded(x, dtype), dtype) for x in synth(2, ends[-1], D, seed=33)]
    cu = torch.tensor(ends, dtype=torch.int32, device="cuda")
    results = []
    for value in (0.0, bad):
        q, k, v, do, dr = (x.clone() for x in ins)
        k[:, ends - 1] = value
        for x in (q, k, v):
            x.requires_grad_()
        o, rem = sb_attn_varlen(q, k, v, cu, max(lengths), zero_start=False)
        _, dk, dv = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
        results.append((o, rem, dk, dv))
    for name, want, got in zip(("o", "rem", "dk", "dv"), *results):
        assert torch.equal(got, want), name


@pytest.mark.parametrize("D,dtype", [(128, torch.bfloat16), (64, torch.float16), (32, torch.bfloat16)])
@pytest.mark.parametrize("fused", [False, True])
def test_blocks_go_from_item_to_item(D, dtype, fused):
    """720 (sequence, head) items, so that every block works on four or five: tile slots, tensor memory and exchange slots are used again,
    phases flip, items come from the counter.  Against the oracle; a second backward from the same workspace gives the same bits (the
    counter starts over)."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    H = 8
    lengths = [int(n) for n in np.random.default_rng(7).permutation(LENGTHS * 6)]
    assert len(lengths) * H >= 4 * torch.cuda.get_device_properties(0).multi_processor_count
    ins = [rounded(x, dtype) for x in synth(H, sum(lengths), D, seed=34)]
    q, k, v, do, dr = (to_dev(x, dtype) for x in ins)
    for x in (q, k, v):
        x.requires_grad_()
    cu = torch.tensor(np.cumsum(lengths), dtype=torch.int32, device="cuda")
    it = 1 / math.sqrt(D)
    o, rem = sb_attn_varlen(q, k, v, cu, max(lengths), zero_start=False, inv_temp=it, fuse_remainder=fused)
    grads = torch.autograd.grad([o, rem], [q, k, v], [do, dr], retain_graph=True)
    again = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
    for x, y in zip(grads, again):
        assert torch.equal(x, y)
    qn, kn, vn, don, drn = ins
    if fused:
        drn = drn + (don.astype(np.float64) * vn).sum(-1)
    want = list(oracle_varlen(qn, kn, vn, don, drn, lengths, it, False))
    if fused:
        want[0] = want[0] + want[1][..., None] * vn
        want[4] = want[4] + want[1][..., None] * don
    got = [x.detach().double().cpu().numpy() for x in (o, rem) + grads]
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    assert_close(("o", "rem", "dq", "dk", "dv"), got, want, TOL_BF16, f"items in turn {D} {dtype} {fused}", out_half_ulp=half_ulp)
