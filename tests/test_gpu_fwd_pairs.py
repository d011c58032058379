"""The forward that works on two query tiles at a time: head dim 128, sequences of one length, at least twelve tiles per SM.  (The first test's packs of
two and more sequences differ too much in length for it: they hold for the other forward as well.)"""
import math

import numpy as np
import pytest
import torch

from oracle import sb_oracle as orc
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
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    if not names:
        pytest.skip("the profiler records no kernels here")
    return {kernel for kernel in ("tc_fwd_pair_kernel", "tc_fwd_kernel") if any(kernel in name for name in names)}


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


def rows(shape, dtype, generator, token_major):
    """N(0, 1) as [..., H, T, D], stored in this order or as [..., T, H, D]."""
    if token_major:
        shape = shape[:-3] + (shape[-2], shape[-3], shape[-1])
    x = torch.randn(shape, generator=generator, device="cuda").to(dtype)
    return (x.transpose(-3, -2) if token_major else x).requires_grad_()


def check_sequences(spans, heads, tensors, grads, it, attend_current, fused, what):
    """The outputs and gradients of some heads of [H, T, ...] tensors against the oracle, sequence by sequence."""
    half_ulp = 2.0 ** -8 if tensors[0].dtype == torch.bfloat16 else 2.0 ** -11
    for start, end in spans:
        for h in heads:
            q, k, v, do, dr, o, rem, dq, dk, dv = (x[h:h + 1, start:end].detach().double().cpu().numpy() for x in tensors + grads)
            if fused:  # out = o + rem v: drem receives do . v, dv receives rem do
                dr = dr + (do * v).sum(-1)
            want = list(oracle_varlen(q, k, v, do, dr, [end - start], it, attend_current))
            if fused:
                want[0] = want[0] + want[1][..., None] * v
                want[4] = want[4] + want[1][..., None] * do
            assert_close(("o", "rem", "dq", "dk", "dv"), (o, rem, dq, dk, dv), want, TOL_BF16, f"{what} head {h} tokens {start}:{end}",
                         out_half_ulp=half_ulp)


@pytest.mark.parametrize("heads,lengths,dtype,token_major,attend_current,fused", [
    (13, [1020, 1030, 1024, 1015] * 4, torch.bfloat16, False, True, False),       # eight and nine tiles, a tile of six rows
    (14, [256] * 64, torch.float16, False, False, True),                            # one pair per sequence
    (9, [300] * 35 + [0] + [300] * 35, torch.bfloat16, False, False, False),        # an empty sequence; the lowest tile alone
    (14, [2048] * 8, torch.bfloat16, True, False, True),
    (14, [2000] * 8, torch.float16, True, True, False),
])
def test_packed_layouts(heads, lengths, dtype, token_major, attend_current, fused):
    from stickbreaking_attention_b200 import sb_attn_varlen
    g = torch.Generator(device="cuda").manual_seed(43)
    T, it = sum(lengths), 1 / math.sqrt(128)
    q, k, v, do = (rows((heads, T, 128), dtype, g, token_major) for _ in range(4))
    dr = torch.randn(heads, T, generator=g, device="cuda").to(dtype)
    ends = np.cumsum(lengths)
    cu = torch.tensor(ends, device="cuda")

    def call():
        return sb_attn_varlen(q, k, v, cu, max(lengths), zero_start=False, attend_current=attend_current, fuse_remainder=fused)
    assert forward_kernels(call) == {"tc_fwd_pair_kernel"}
    o, rem = call()
    grads = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
    spans = [(int(ends[i]) - lengths[i], int(ends[i])) for i in (0, 1, len(lengths) // 2 + 1, len(lengths) - 1)]
    check_sequences(spans, (0, heads - 1), (q, k, v, do, dr), (o, rem) + grads, it, attend_current, fused, "packed")


@pytest.mark.parametrize("batch,heads,tokens,dtype,token_major,attend_current,fused", [
    (8, 28, 1024, torch.float16, True, False, True),
    (8, 28, 1000, torch.bfloat16, False, True, False),
    (5, 30, 1537, torch.bfloat16, True, False, False),
])
def test_batched_layouts(batch, heads, tokens, dtype, token_major, attend_current, fused):
    from stickbreaking_attention_b200 import sb_attn
    g = torch.Generator(device="cuda").manual_seed(47)
    q, k, v, do = (rows((batch, heads, tokens, 128), dtype, g, token_major) for _ in range(4))
    dr = torch.randn(batch, heads, tokens, generator=g, device="cuda").to(dtype)

    def call():
        return sb_attn(q, k, v, attend_current=attend_current, fuse_remainder=fused)
    assert forward_kernels(call) == {"tc_fwd_pair_kernel"}
    o, rem = call()
    grads = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
    for b in (0, batch - 1):
        check_sequences([(0, tokens)], (0, 3, heads - 1), tuple(x[b] for x in (q, k, v, do, dr)), tuple(x[b] for x in (o, rem) + grads),
                        1 / math.sqrt(128), attend_current, fused, f"batched entry {b}")


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_what_a_neighbour_holds_stays_there(value):
    """Tiles at a sequence's end hold rows of the next sequence: whatever these are, the results are the same bits."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    H, n, L = 14, 16, 1000
    g = torch.Generator(device="cuda").manual_seed(53)
    x = [torch.randn(H, n * L, 128, generator=g, device="cuda").bfloat16() for _ in range(3)]
    cu = torch.arange(1, n + 1, device="cuda") * L

    def call(q, k, v):
        with torch.no_grad():
            return sb_attn_varlen(q, k, v, cu, L, zero_start=False)
    assert forward_kernels(lambda: call(*x)) == {"tc_fwd_pair_kernel"}
    want = call(*x)
    for t in x:
        t[:, 5 * L:6 * L] = value
    got = call(*x)
    for a, b in zip(got, want):
        assert torch.equal(a[:, :5 * L], b[:, :5 * L]) and torch.equal(a[:, 6 * L:], b[:, 6 * L:])


def test_eight_heads_of_8x4096():
    """Eight sequences of 4096 tokens with heads enough for pairs: some (head, sequence) in full."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    H, L, n = 8, 4096, 8
    g = torch.Generator(device="cuda").manual_seed(59)
    q, k, v, do = (rows((H, n * L, 128), torch.bfloat16, g, False) for _ in range(4))
    dr = torch.randn(H, n * L, generator=g, device="cuda").bfloat16()
    cu = torch.arange(1, n + 1, device="cuda", dtype=torch.int32) * L

    def call():
        return sb_attn_varlen(q, k, v, cu, L, zero_start=False)
    assert forward_kernels(call) == {"tc_fwd_pair_kernel"}
    o, rem = call()
    grads = torch.autograd.grad([o, rem], [q, k, v], [do, dr])
    for h, s in ((0, 0), (7, 7), (3, 4)):
        check_sequences([(s * L, (s + 1) * L)], (h,), (q, k, v, do, dr), (o, rem) + grads, 1 / math.sqrt(128), False, False, "8 x 4096")


@pytest.mark.parametrize("heads,tokens", [(28, 8192), (4, 65536)])
def test_rows_of_one_long_sequence(heads, tokens):
    """o, rem and dq on row slabs against the oracle with all keys to their left (257 and more steps of a pair in the longer one)."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    g = torch.Generator(device="cuda").manual_seed(61)
    it = 1 / math.sqrt(128)
    q, k, v, do = ((0.5 * torch.randn(heads, tokens, 128, generator=g, device="cuda")).bfloat16().requires_grad_() for _ in range(4))
    dr = torch.randn(heads, tokens, generator=g, device="cuda").bfloat16()
    cu = torch.tensor([tokens], device="cuda")

    def call():
        return sb_attn_varlen(q, k, v, cu, tokens, zero_start=False)
    assert forward_kernels(call) == {"tc_fwd_pair_kernel"}
    o, rem = call()
    dq, = torch.autograd.grad([o, rem], [q], [do, dr])
    for h in (0, heads - 1):
        Q, K, V, DO, DR = (x[h:h + 1].detach().double().cpu().numpy() for x in (q, k, v, do, dr))
        for lo in (0, tokens // 2 - 100, tokens - 256):
            want = orc.sb_rows_fwd(Q, K, V, 0, lo, lo + 256, it) + (orc.sb_rows_dq(Q, K, V, DO, DR, 0, lo, lo + 256, it),)
            got = [x[h:h + 1, lo:lo + 256].detach().double().cpu().numpy() for x in (o, rem, dq)]
            assert_close(("o", "rem", "dq"), got, want, TOL_BF16, f"head {h} rows {lo}", out_half_ulp=2.0 ** -8)
