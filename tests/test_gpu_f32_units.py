"""The tcgen05 kernels of float32 precision: rows that loads take in units of four, two or one elements (by alignment and strides), and lengths
on both sides of their steps of 64 keys, chunks of 32 queries and tiles of 128."""
import math

import numpy as np
import pytest
import torch

from util import TOL_BF16, TOL_F32, assert_close, oracle_varlen, rounded, synth, to_dev

pytestmark = pytest.mark.gpu

LENGTHS = [1, 33, 63, 97, 129, 161, 257, 1121, 2049, 3900]  # 781 on average: these kernels at every head dim up to 64


def _placed(x, unit):
    """The same values at an address and with a row stride that are multiples of `unit` elements and of no more."""
    H, T, D = x.shape
    buf = torch.empty(H * T * (D + 4) + 8, dtype=x.dtype, device=x.device)
    out = buf[unit:].as_strided((H, T, D), (T * (D + unit), D + unit, 1))
    return out.copy_(x).detach()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,unit", [(64, 4), (64, 2), (64, 1), (36, 4), (50, 2), (33, 1), (16, 2), (1, 1)])
def test_units_and_lengths(dtype, D, unit):
    from stickbreaking_attention_b200 import sb_attn_varlen
    ins = [rounded(x, dtype) for x in synth(2, sum(LENGTHS), D, seed=61)]
    q, k, v, do = (_placed(to_dev(x, dtype), unit) for x in ins[:4])
    for x in (q, k, v):
        x.requires_grad_()
    cu = torch.tensor(np.cumsum(LENGTHS), device="cuda")
    o, rem = sb_attn_varlen(q, k, v, cu, max(LENGTHS), zero_start=False)
    got = [o, rem, *torch.autograd.grad([o, rem], [q, k, v], [do, to_dev(ins[4], dtype)])]
    want = oracle_varlen(*ins, LENGTHS, 1 / math.sqrt(D), False)
    # float32: a few units of 2^-24 of sums that reach 5; 16-bit types: the output format
    tol = TOL_F32 if dtype == torch.float32 else TOL_BF16
    assert_close(("o", "rem", "dq", "dk", "dv"), [x.detach().double().cpu().numpy() for x in got], want, tol, f"{dtype} {D} {unit}", out_half_ulp=2**-8 if dtype == torch.bfloat16 else 0.0)
