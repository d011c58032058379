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


def forward_kernels(call):
    """Names of the forward kernels that `call` launches."""
    from torch.profiler import ProfilerActivity, profile
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return {name for e in prof.events() for name in ("tc_fwd_pair_kernel", "tc_fwd_kernel") if name in e.name}


@pytest.mark.parametrize("heads,tokens", [(16, 16384), (33, 8192), (7, 32768)])  # groups of 5, 8 and 2 heads, one head in the first group
def test_heads_that_do_not_fill_their_groups(heads, tokens):
    """Every head is worked on once: each against the same head in a call of few heads, which works on single tiles; both round their
    16-bit weights and results from the same float32 sums, so they differ by a unit in the last place of results and the error of the weights
    (2^-8 of each, in a weighted mean of N(0, 1) values: far below the bar)."""
    from stickbreaking_attention_b200 import sb_attn
    g = torch.Generator(device="cuda").manual_seed(heads)
    q, k, v = (torch.randn(1, heads, tokens, 128, generator=g, device="cuda").bfloat16() for _ in range(3))
    with torch.no_grad():
        assert forward_kernels(lambda: sb_attn(q, k, v)) == {"tc_fwd_pair_kernel"}
        o, rem = sb_attn(q, k, v)
        few = max(1, 8 * torch.cuda.get_device_properties(0).multi_processor_count * 128 // tokens // 2)
        for h in range(0, heads, few):
            part = [x[:, h:h + few] for x in (q, k, v)]
            assert forward_kernels(lambda: sb_attn(*part)) == {"tc_fwd_kernel"}
            want_o, want_rem = sb_attn(*part)
            assert torch.all((o[:, h:h + few] - want_o).abs() <= 2.0 ** -7 * want_o.abs() + TOL_BF16)
            assert torch.all((rem[:, h:h + few].float() - want_rem.float()).abs() <= 2.0 ** -7 * want_rem.float().abs() + 1e-6)


def test_a_head_more_costs_a_head_more():
    """Sixteen heads of 16 384 tokens go as groups of 1, 5, 5 and 5.  With the single head last, its longest pair (two rows of 128 tiles, about
    4.5 times a head's share of all SMs) ends the kernel alone: 1.25 times the time of fifteen heads.  With it first the ratio is about 16 / 15;
    the bar lies between the two."""
    from stickbreaking_attention_b200 import sb_attn
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(1, 16, 16384, 128, generator=g, device="cuda").bfloat16() for _ in range(3))

    def fastest(heads):
        part = [x[:, :heads] for x in (q, k, v)]
        times = []
        with torch.no_grad():
            for i in range(8):
                start, end = (torch.cuda.Event(enable_timing=True) for _ in range(2))
                start.record()
                for _ in range(3):
                    sb_attn(*part)
                end.record()
                end.synchronize()
                times.append(start.elapsed_time(end))
        return min(times[2:])
    fifteen, sixteen = fastest(15), fastest(16)
    assert sixteen <= 1.18 * fifteen, (fifteen, sixteen)


@pytest.mark.parametrize("heads,lengths,pairs", [
    (32, [8192], True),
    (12, [8192] * 4, True),
    (8, [65536], True),
    (17, [16384], True),
    (16, [256] * 64, True),
    (16, [1020, 1030, 1024, 1015] * 4, True),  # within 1/64 of the average
    (6, [8192], False),                         # 2.6 tiles per SM
    (10, [256] * 64, False),                    # 8.6 tiles per SM
    (20, [870, 1130, 1000, 1100, 900] * 3, False),   # lengths that differ: 0.97 ... 1.0 times as fast in pairs
    (32, [2943, 3503, 2192, 1807, 3696, 649, 1594], False),
    (28, [257] * 31, False),                    # 0.99: a row in the last tile of three
    (128, [2048], False),                       # 0.945: eight heads have too few long pairs for all SMs
    (56, [4096], False),                        # 0.92
])
def test_calls_that_go_in_pairs(heads, lengths, pairs):
    """The rule takes what two query tiles at a time are faster at, and nothing that they are slower at."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the cases are those of 148 SMs")
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(heads, sum(lengths), 128, generator=g, device="cuda").bfloat16() for _ in range(3))
    cu = torch.tensor(np.cumsum(lengths), device="cuda")
    with torch.no_grad():
        ran = forward_kernels(lambda: sb_attn_varlen(q, k, v, cu, max(lengths), zero_start=False))
    assert ran == {"tc_fwd_pair_kernel" if pairs else "tc_fwd_kernel"}
