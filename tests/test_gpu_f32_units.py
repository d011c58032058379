"""The tcgen05 kernels of float32 precision: rows that loads take in units of four, two or one elements (by alignment and strides), lengths
on both sides of their steps of 64 keys, chunks of 32 queries and tiles of 128, and the precision of their sums and of their sigmoid."""
import math

import numpy as np
import pytest
import torch

from util import TOL_F32, assert_close, oracle_varlen, rounded, run_varlen, synth, to_dev

pytestmark = pytest.mark.gpu

NAMES = ("o", "rem", "dq", "dk", "dv")
LENGTHS = [1, 33, 63, 97, 129, 161, 257, 1121, 2049, 3900]  # 781 on average: these kernels at every head dim up to 64
# 16-bit results are float32 sums rounded once: on top of the float32 bar (a few units of 2^-24 of sums that reach 5) half a unit in the last place
HALF_ULP = {torch.float32: 0.0, torch.float16: 2**-11, torch.bfloat16: 2**-8}


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
    assert_close(NAMES, [x.detach().double().cpu().numpy() for x in got], want, TOL_F32, f"{dtype} {D} {unit}", out_half_ulp=HALF_ULP[dtype])


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 20), (torch.float16, 50), (torch.bfloat16, 16)])
def test_attend_current_and_lost_terms(dtype, D):
    """Queries that see their own key; and the bar tells two terms from one: the same sums over inputs cut to one bf16 term exceed it."""
    lengths = [1, 900, 65, 2049, 833, 1121]
    ins = [rounded(x, dtype) for x in synth(1, sum(lengths), D, seed=62)]
    scale = 1 / math.sqrt(D)
    got = run_varlen(*ins, lengths, scale, True, dtype)
    want = oracle_varlen(*ins, lengths, scale, True)
    assert_close(NAMES, got, want, TOL_F32, f"{dtype} {D}", out_half_ulp=HALF_ULP[dtype])
    if dtype != torch.bfloat16:
        worse = oracle_varlen(*[rounded(x, torch.bfloat16) for x in ins], lengths, scale, True)
        for name, g, w in zip(NAMES, worse, want):
            assert (np.abs(g - w) - np.abs(w) * HALF_ULP[dtype]).max() > TOL_F32, name


@pytest.mark.parametrize("D", [64, 24])
def test_norm_of_the_error(D):
    """float32: the norm of the error against that of the result.  Three terms and sums of at most 64 products from zero are off by about 2^-23
    (1.2e-7; 0.8e-7 to 1.6e-7 measured); the bar is four times that, what a loss of two bits makes of it."""
    lengths = [1121, 2049]
    ins = synth(2, sum(lengths), D, seed=63)
    got = run_varlen(*ins, lengths, 1 / math.sqrt(D), False, torch.float32)
    want = oracle_varlen(*ins, lengths, 1 / math.sqrt(D), False)
    for name, g, w in zip(NAMES, got, want):
        err = np.linalg.norm(g - w) / np.linalg.norm(w)
        print(f"norm of the error, head dim {D}, {name}: {err:.2e}")
        assert err <= 2**-21, (name, err)


def test_sigmoid():
    """The first row of a sequence with attend_current: o = sigmoid(x) v, rem = 1 - sigmoid(x), both with full relative precision (an exponential of
    at most 2 ulp, a reciprocal after one step of Newton's method, a product: 5 ulp), down to the smallest normal numbers."""
    from stickbreaking_attention_b200 import sb_attn
    x = torch.linspace(-86, 86, 4097)
    x = torch.cat([x, torch.linspace(-1e-3, 1e-3, 4096)]).float()
    q = torch.zeros(x.numel(), 1, 128, 33, device="cuda")
    k, v = torch.zeros_like(q), torch.zeros_like(q)
    q[:, 0, 0, 0] = x.cuda()
    k[:, 0, 0, 0] = 1
    v[:, 0, 0, 0] = 1
    with torch.no_grad():
        o, rem = sb_attn(q, k, v, inv_temp=1.0, attend_current=True)
    x = x.double()
    for got, want in ((o[:, 0, 0, 0], 1 / (1 + torch.exp(-x))), (rem[:, 0, 0], 1 / (1 + torch.exp(x)))):
        assert ((got.cpu().double() - want).abs() / want).max() <= 5 * 2**-23
