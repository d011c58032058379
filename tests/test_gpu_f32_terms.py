"""The kernels of float32 precision at head dims and lengths where their tiles end: rows read in units of one, two or four
elements, head dims on both sides of the tile widths, sequence ends on both sides of 32 and 64."""
import math

import numpy as np
import pytest
import torch

from util import TOL_BF16, TOL_F32, assert_close, oracle_varlen, rounded, run_varlen, synth, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D", [(torch.float32, 33), (torch.float32, 8), (torch.float32, 100), (torch.float32, 128), (torch.bfloat16, 33),
                                     (torch.bfloat16, 17), (torch.float16, 100), (torch.float16, 66)])
@pytest.mark.parametrize("attend_current", [False, True])
def test_edges_against_oracle(dtype, D, attend_current):
    lengths = [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 193]
    ins = [rounded(x, dtype) for x in synth(2, sum(lengths), D, seed=51)]
    got = run_varlen(*ins, lengths, 1 / math.sqrt(D), attend_current, dtype)
    want = oracle_varlen(*ins, lengths, 1 / math.sqrt(D), attend_current)
    # float32: a few units of 2^-24 of sums that reach 5; 16-bit types: the output format
    assert_close(("o", "rem", "dq", "dk", "dv"), got, want, TOL_F32 if dtype == torch.float32 else TOL_BF16, f"{dtype} {D}")


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 20), (torch.bfloat16, 50), (torch.bfloat16, 16), (torch.float16, 33)])
def test_many_blocks_against_oracle(dtype, D):
    """Enough (sequence, tile, head) blocks for the dk/dv form with two blocks per SM: lengths on both sides of its steps of 32 queries."""
    lengths = [1, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 161, 193] * 2
    ins = [rounded(x, dtype) for x in synth(16, sum(lengths), D, seed=52)]
    got = run_varlen(*ins, lengths, 1 / math.sqrt(D), False, dtype)
    want = oracle_varlen(*ins, lengths, 1 / math.sqrt(D), False)
    assert_close(("o", "rem", "dq", "dk", "dv"), got, want, TOL_F32 if dtype == torch.float32 else TOL_BF16, f"{dtype} {D}")


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 100), (torch.bfloat16, 50), (torch.float16, 16)])
@pytest.mark.parametrize("copies", [1, 24])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_rows_behind_a_sequence_see_no_key(dtype, D, copies, bad):
    """The last key of every sequence is visible to no query: whatever its k holds, o, rem, dk and dv are the same bits, in both forms
    of dk/dv (`copies`: enough blocks for the one with two blocks per SM)."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    lengths = [1, 31, 33, 63, 65, 100, 129] * copies
    ends = np.cumsum(lengths)
    ins = [to_dev(rounded(x, dtype), dtype) for x in synth(2, ends[-1], D, seed=53)]
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
