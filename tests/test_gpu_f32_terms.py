"""The kernels of float32 precision at head dims and lengths where their tiles end: rows read in units of one, two or four
elements, head dims on both sides of the tile widths, sequence ends on both sides of 32 and 64."""
import math

import pytest
import torch

from util import TOL_BF16, TOL_F32, assert_close, oracle_varlen, rounded, run_varlen, synth

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
