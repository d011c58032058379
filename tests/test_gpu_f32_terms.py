"""The kernels of float32 precision at head dims and lengths where their tiles end: rows read in units of one, two or four
elements, head dims on both sides of the tile widths, sequence ends on both sides of 32 and 64; and values that do not divide into terms.
LONG brings head dims up to 64 to the kernels on tcgen05, shorter packs to those on warp-level matrix instructions."""
import math

import numpy as np
import pytest
import torch

from util import TOL_BF16, TOL_F32, assert_close, oracle_varlen, rounded, run_varlen, synth, to_dev

pytestmark = pytest.mark.gpu

LONG = [900, 700, 810]  # 803 on average; last tiles of 4, 60 and 42 rows

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
@pytest.mark.parametrize("pack", [[1, 31, 33, 63, 65, 100, 129], [1, 31, 33, 63, 65, 100, 129] * 24, [897, 800, 961, 1000]])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_rows_behind_a_sequence_see_no_key(dtype, D, pack, bad):
    """The last key of every sequence is visible to no query: whatever its k holds, o, rem and dv are the same bits, in both forms of
    dk/dv on warp-level instructions (the second pack: enough blocks for the one with two blocks per SM) and on tcgen05, and dk the same but for the rounding of the prefix sums that the
    dq kernel leaves it (dq itself is NaN, zero times k, and formed again by multiply-adds)."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    lengths = pack
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
        results.append((o, rem, dv, dk))
    for name, want, got in zip(("o", "rem", "dv"), *results):
        assert torch.equal(got, want), name
    want, got = (r[3].double() for r in results)
    assert (got - want).abs().max() <= (1e-6 if dtype == torch.float32 else 1e-2) * want.abs().max()


@pytest.mark.parametrize("dtype,D,length", [(torch.float32, 64, 140), (torch.bfloat16, 50, 257), (torch.float16, 20, 320), (torch.bfloat16, 18, 385),
                                            (torch.float32, 16, 800), (torch.bfloat16, 9, 800), (torch.bfloat16, 18, 320)])
@pytest.mark.parametrize("ragged", [False, True])
def test_forward_and_backward_choose_apart(dtype, D, length, ragged):
    """Equal lengths whose last tile is at most half full, more than three blocks per SM: the forward mostly runs on tcgen05 there and the backward on
    warp-level instructions, over the carries that the forward has left.  `ragged`: the same average, on tcgen05 both ways."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    lengths = [length - 100, length + 101, length] if ragged else [length] * 3
    ins = [rounded(x, dtype) for x in synth(2, sum(lengths), D, seed=57)]
    heads = 148 * 3 // 6 + 1  # the two heads again and again: three sequences of at least two tiles each
    tensors = [to_dev(x, dtype).repeat(heads, *[1] * (x.ndim - 1)) for x in ins]
    for x in tensors[:3]:
        x.requires_grad_()
    q, k, v, do, dr = tensors
    o, rem = sb_attn_varlen(q, k, v, torch.tensor(np.cumsum(lengths), device="cuda"), max(lengths), zero_start=False)
    results = (o, rem, *torch.autograd.grad([o, rem], [q, k, v], [do, dr]))
    for x in results:
        assert torch.equal(x[:-2], x[2:])  # whatever block a head's tile got
    got = [x[:2].detach().double().cpu().numpy() for x in results]
    want = oracle_varlen(*ins, lengths, 1 / math.sqrt(D), False)
    half_ulp = {torch.float32: 0.0, torch.float16: 2**-11, torch.bfloat16: 2**-8}[dtype]  # of the results, which are float32 sums rounded once
    assert_close(("o", "rem", "dq", "dk", "dv"), got, want, TOL_F32, f"{dtype} {D}", out_half_ulp=half_ulp)


def _dense(q, k, v, do, dr, lengths, scale):
    """The operator and its gradients as dense float64 sums in which an infinity is an infinity (products of 1 - beta, no logarithms)."""
    out = [np.zeros(x, np.float64) for x in (q.shape, dr.shape, q.shape, q.shape, q.shape)]
    with np.errstate(all="ignore"):
        for h in range(q.shape[0]):
            for end, n in zip(np.cumsum(lengths), lengths):
                at = np.s_[h, end - n:end]
                Q, K, V, G, R = (np.asarray(x, np.float64)[at] for x in (q, k, v, do, dr))
                s = Q @ K.T * scale
                seen = np.tril(np.ones((n, n), bool), -1)
                beta, r = np.where(seen, 1 / (1 + np.exp(-s)), 0), np.where(seen, 1 / (1 + np.exp(s)), 1)
                right = np.cumprod(np.concatenate([r, np.ones((n, 1))], 1)[:, ::-1], 1)[:, ::-1]  # [:, j]: over the keys >= j
                A = beta * right[:, 1:]
                A[A < 2.0 ** -100] = 0  # may be zero in float32: what it makes of an infinity is left open
                g = A * (G @ V.T - R[:, None])
                ds = (g - beta * np.cumsum(g, 1)) * scale
                for x, y in zip(out, (A @ V, right[:, 0], ds @ K, ds.T @ Q, A.T @ G)):
                    x[at] = y
    return out


@pytest.mark.parametrize("dtype,D", [(torch.float32, 64), (torch.float32, 100), (torch.float32, 16), (torch.float16, 50), (torch.bfloat16, 50)])
@pytest.mark.parametrize("pack", [[150, 40], [150, 40] * 24, LONG])
@pytest.mark.parametrize("what,value,checked", [
    ("k", np.inf, "o rem dk dv"), ("q", -np.inf, "o rem dq dv"), ("v", np.inf, "o rem dv"), ("do", -np.inf, "o rem dv"),  # one element
    ("v", np.finfo(np.float32).max, "o rem dv"), ("k", np.finfo(np.float32).min, "o rem dk dv"),
    ("v", None, "o rem"), ("do", None, "dq dk dv"),  # the whole tensor (and dr with do) times 1e-36
])
def test_values_that_terms_do_not_hold(dtype, D, pack, what, value, checked):
    """Infinities, float32's largest values (beyond bf16's) and magnitudes whose later terms would lie below bf16's smallest, against
    dense float64 sums: finite where those are, the same infinities, no bits lost (the packs: both forms of dk/dv on
    warp-level instructions, and the kernels on tcgen05, with a bad element in each half of a 128-row tile and in a last tile of 4 rows)."""
    if dtype == torch.float16 and (value is None or np.isfinite(value)):
        pytest.skip("beyond the range of float16")
    lengths = pack
    q, k, v, do, dr = synth(2, sum(lengths), D, seed=54)
    if value is None:
        for x in {"v": [v], "do": [do, dr]}[what]:
            x *= np.float32(1e-36)
    else:
        for pos in (40, 130, 200, 898) if pack == LONG else (40, 130):
            {"q": q, "k": k, "v": v, "do": do}[what][0, pos, 3] = value
    ins = [rounded(x, dtype) for x in (q, k, v, do, dr)]
    scale = 1 / math.sqrt(D)
    got = run_varlen(*ins, lengths, scale, False, dtype)
    want = _dense(*ins, lengths, scale)
    for name, g, w in zip(("o", "rem", "dq", "dk", "dv"), got, want):
        if name not in checked.split():
            continue
        finite, inf = np.isfinite(w), np.isinf(w)
        assert np.isfinite(g[finite]).all(), name
        assert np.array_equal(g[inf], w[inf]), name
        # relative to the largest result (float32: sums of up to 900 products, whose errors grow with the root of their number; 16-bit types: rounding of the result)
        most = np.abs(w[finite]).max()
        err = np.abs(g[finite] - w[finite]).max() / most
        assert err <= (1e-5 if dtype == torch.float32 else 1e-2), (name, err)


@pytest.mark.parametrize("pack", [[150, 40], LONG])
@pytest.mark.parametrize("D", [64, 40, 16])
@pytest.mark.parametrize("what,result", [("v", "o"), ("k", "dq"), ("q", "dk"), ("do", "dv")])
def test_tiny_columns_among_ordinary_ones(pack, D, what, result):
    """Two of every eight columns times 1e-36: results below 2^-100 beside ordinary ones lose no bits either."""
    names = ("o", "rem", "dq", "dk", "dv")
    ins = dict(zip(("q", "k", "v", "do", "dr"), synth(2, sum(pack), D, seed=56)))
    tiny = np.arange(D) % 8 < 2
    ins[what][..., tiny] *= np.float32(1e-36)
    scale = 1 / math.sqrt(D)
    got = dict(zip(names, run_varlen(*ins.values(), pack, scale, False, torch.float32)))[result]
    want = dict(zip(names, _dense(*ins.values(), pack, scale)))[result]
    for columns in (tiny, ~tiny):
        g, w = got[..., columns], want[..., columns]
        assert np.abs(g - w).max() <= 1e-5 * np.abs(w).max()  # as above


def test_more_blocks_than_one_grid_axis_takes():
    """513 heads x 2^21 sequences (all but two of them empty): 2.15e9 blocks, more than 2^31 - 1."""
    from stickbreaking_attention_b200 import sb_attn_varlen
    H, T, D, S = 513, 64, 16, 1 << 21
    q = torch.randn(H, T, D, device="cuda", generator=torch.Generator("cuda").manual_seed(55))
    cu = torch.full((S,), T, dtype=torch.int32, device="cuda")
    cu[:4] = torch.tensor([0, 7, 7, T])
    with torch.no_grad():
        want = sb_attn_varlen(q, q, q, torch.tensor([7, T], device="cuda"), T, zero_start=False)
        got = sb_attn_varlen(q, q, q, cu, T, zero_start=False)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
