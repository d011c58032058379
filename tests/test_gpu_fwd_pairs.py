"""The forward that works on two query tiles at a time: head dim 128, sequences of about the same length, at least twelve tiles per SM."""
import math

import numpy as np
import pytest
import torch

from util import TOL_BF16, assert_close, oracle_varlen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths,dtype,attend_current,fused", [
    ([513, 640, 600, 576, 529, 625], torch.bfloat16, False, False),  # five tiles each: the lowest stands alone; ends on and off multiples of 16
    ([513, 640, 600, 576, 529, 625], torch.float16, True, True),
    ([1024, 1025, 900, 1100], torch.float16, False, False),          # even and odd numbers of tiles, a tile of one row
    ([1024, 1025, 900, 1100], torch.bfloat16, True, True),
    ([2049], torch.bfloat16, False, True),
])
def test_pairs_of_tiles_against_oracle(lengths, dtype, attend_current, fused):
    """Forward and the gradients that follow from its carries, with NaN in the pad behind the last sequence."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    D, T, pad = 128, sum(lengths), 7
    tiles = sum(-(-n // 128) for n in lengths)
    H = -(-12 * torch.cuda.get_device_properties(0).multi_processor_count // tiles)
    g = torch.Generator(device="cuda").manual_seed(41)
    q, k, v, do = (torch.randn(H, T + pad, D, generator=g, device="cuda").to(dtype) for _ in range(4))
    dr = torch.randn(H, T + pad, generator=g, device="cuda").to(dtype)
    for x in (q, k, v, do):
        x[:, T:] = float("nan")
        x.requires_grad_(x is not do)
    cu = torch.tensor(np.cumsum(lengths), device="cuda")
    it = 1 / math.sqrt(D)

    def call():
        return sb_attn_varlen(q, k, v, cu, max(lengths), zero_start=False, inv_temp=it, attend_current=attend_current, fuse_remainder=fused)
    o, rem = call()
    grads = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
    with torch.no_grad():  # without carries: the same bits
        o2, rem2 = call()
    assert torch.equal(o[:, :T], o2[:, :T]) and torch.equal(rem, rem2)
    assert torch.all(rem[:, T:] == 0)
    heads = [0, H // 2, H - 1]
    qn, kn, vn, don = (x[heads, :T].detach().float().cpu().numpy() for x in (q, k, v, do))
    drn = dr[heads, :T].float().cpu().numpy()
    if fused:  # out = o + rem v: drem receives do . v, dv receives rem do
        drn = drn + (don.astype(np.float64) * vn).sum(-1)
    want = list(oracle_varlen(qn, kn, vn, don, drn, lengths, it, attend_current))
    if fused:
        want[0] = want[0] + want[1][..., None] * vn
        want[4] = want[4] + want[1][..., None] * don
    got = [x[heads, :T].detach().double().cpu().numpy() for x in (o, rem) + grads]
    half_ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11  # what storing the exact result in the output type costs
    assert_close(("o", "rem", "dq", "dk", "dv"), got, want, TOL_BF16, f"pairs {lengths} {dtype} {fused}", out_half_ulp=half_ulp)
