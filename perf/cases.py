"""Performance cases of the stick-breaking attention operators: what users of this package have them do.

Every case is one call through the public entry points ``sb_attn_varlen`` (packed [H, T, D]) or ``sb_attn`` (batched
[B, H, T, D]): the forward alone under ``torch.no_grad`` (evaluation, prefill) or forward and backward through autograd
(training).  The fields of a case:

  layout       'packed' or 'batched'
  train        True: forward + backward; False: forward without gradients
  dtype        'bf16', 'f16', 'f32'
  heads, dim   attention heads and head dim
  lengths      packed: the sequence lengths as text, "128,192,192"; batched: "BxT"
  dist         'normal': N(0, 1) inputs; 'half': 0.5 N(0, 1) (long context); 'negative': logits of negative mean, as in the
               tests of the operator (0.25 (N + 1) queries against 0.25 (N - 1) keys)
  token_major  the tensors are stored as [T, H, D] ([B, T, H, D]) and passed as permuted views, the way a projection leaves them
  fuse         ask for out = o + rem * v (what callers form next) instead of o
  current      attend_current: a query also sees its own key
  bare         packed: cu_seqlens with its leading zero and no max_seqlens, the shortest way to call the operator
               (otherwise sequence ends alone and max_seqlens given)
"""
import math

import torch

from stickbreaking_attention_b200 import sb_attn, sb_attn_varlen

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
BYTES = {"bf16": 2, "f16": 2, "f32": 4}


def _case(layout, train, dtype, heads, dim, lengths, dist="normal", token_major=False, fuse=False, current=False, bare=False):
    return dict(layout=layout, train=train, dtype=dtype, heads=heads, dim=dim, lengths=lengths, dist=dist,
                token_major=token_major, fuse=fuse, current=current, bare=bare)


def listed():
    return [
        # the smallest call that makes sense: one layer of a small model evaluates three short prompts
        dict(_case("packed", False, "bf16", 4, 64, "37,64,27"), name="eval-tiny"),
        # correctness-scale training step in float32: 4 heads, 512 tokens in three sequences
        dict(_case("packed", True, "f32", 4, 64, "128,192,192"), name="train-f32-512"),
        # the batched layout at the odd sizes of the operator's own tests: 500 tokens, head dim 50
        dict(_case("batched", True, "bf16", 8, 50, "4x500", dist="negative"), name="train-batched-d50"),
        # a small fine-tuning micro-batch: 2048 tokens in ragged documents, each query also sees its own key
        dict(_case("packed", True, "bf16", 8, 64, "611,90,333,402,127,485", current=True), name="train-small"),
        # float16 batched training at a length that is no multiple of a tile, straight from a [B, T, H, D] projection
        dict(_case("batched", True, "f16", 16, 64, "2x1000", token_major=True), name="train-batched-f16"),
        # float32 training at an ordinary size (numerically sensitive layers, reference runs)
        dict(_case("packed", True, "f32", 8, 64, "1024,700,1324,1048"), name="train-f32-4096"),
        # the shortest way to call the packed operator, token-major tensors and the fused output: 12 heads, 8192 tokens
        dict(_case("packed", True, "bf16", 12, 128, "3000,1500,2692,1000", token_major=True, fuse=True, bare=True), name="train-bare-fused"),
        # many short documents in one pack: bound by memory rather than by arithmetic
        dict(_case("packed", True, "bf16", 32, 128, ",".join(["128"] * 512)), name="train-short-docs"),
        # prefill of one 8192-token prompt
        dict(_case("packed", False, "bf16", 32, 128, "8192"), name="prefill-8192"),
        # the ordinary training pack: 32 heads, 16384 tokens in sequences of 649 ... 3696
        dict(_case("packed", True, "bf16", 32, 128, "2943,3503,2192,1807,3696,649,1594"), name="train-pack-16384"),
        # the layout and shape of the operator's benchmark: four sequences of 8192 tokens, 12 heads, token-major, out = o + rem v
        dict(_case("packed", True, "bf16", 12, 128, "8192,8192,8192,8192", token_major=True, fuse=True), name="train-4x8192"),
        # long context: one sequence of 65536 tokens
        dict(_case("packed", True, "bf16", 8, 128, "65536", dist="half"), name="train-long-65536"),
    ]


# The largest of everything that a drawn case may reach: the long-context case's arithmetic, the short-document case's elements.
MOST_FLOPS = 3.0e13
MOST_ELEMENTS = 32 * 65536 * 128
# float32 inputs and odd head dims are used at test and fine-tuning scale
MOST_FLOPS_SMALL = 1.2e11


def draw(rng):
    while True:
        train = rng.random() < 0.7
        dtype = rng.choice(["bf16", "bf16", "bf16", "f16", "f32"])
        dim = rng.choice([128, 128, 128, 64, 64, 64, 32, 50, 16])
        heads = rng.choice([1, 2, 3, 4, 6, 8, 12, 16, 24, 32])
        small = dtype == "f32" or dim in (16, 50)
        tokens = int(round(math.exp(rng.uniform(math.log(100), math.log(8192 if small else 65536)))))
        flags = dict(token_major=rng.random() < 0.3, fuse=rng.random() < 0.25, current=rng.random() < 0.2,
                     dist=rng.choice(["normal", "normal", "negative"]))
        if rng.random() < 0.3:
            batch = min(rng.choice([1, 2, 3, 4, 8, 16]), tokens)
            case = _case("batched", train, dtype, heads, dim, "%dx%d" % (batch, max(1, tokens // batch)), **flags)
        else:
            mean = math.exp(rng.uniform(math.log(64), math.log(max(65, tokens))))
            lens, left = [], tokens
            while left > 0:
                n = min(left, max(1, int(round(mean * math.exp(rng.gauss(0, 0.6))))))
                lens.append(n)
                left -= n
            case = _case("packed", train, dtype, heads, dim, ",".join(map(str, lens)), bare=rng.random() < 0.2, **flags)
        if work(case)["flops"] <= (MOST_FLOPS_SMALL if small else MOST_FLOPS) and heads * tokens * dim <= MOST_ELEMENTS:
            return case


def _sizes(case):
    """(batch, tokens per batch entry, sequence lengths)"""
    if case["layout"] == "batched":
        batch, tokens = (int(x) for x in case["lengths"].split("x"))
        return batch, tokens, [tokens] * batch
    lens = [int(x) for x in case["lengths"].split(",")]
    return 1, sum(lens), lens


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    batch, tokens, lens = _sizes(case)
    heads, dim, dtype = case["heads"], case["dim"], DTYPES[case["dtype"]]
    packed = case["layout"] == "packed"
    lead = () if packed else (batch,)

    def rows(mean=0.0, scale=1.0):
        shape = lead + ((tokens, heads, dim) if case["token_major"] else (heads, tokens, dim))
        x = torch.randn(shape, generator=g, device="cuda", dtype=dtype)
        if mean or scale != 1.0:
            x.add_(mean).mul_(scale)
        return x.transpose(-3, -2) if case["token_major"] else x

    if case["dist"] == "negative":
        q, k, v = rows(1.0, 0.25), rows(-1.0, 0.25), rows(0.0, 0.25)
    else:
        s = 0.5 if case["dist"] == "half" else 1.0
        q, k, v = rows(0.0, s), rows(0.0, s), rows(0.0, s)
    state = dict(case=case, q=q, k=k, v=v)
    if packed:
        ends = torch.tensor(lens, device="cuda").cumsum(0)
        state["cu"] = torch.cat([ends.new_zeros(1), ends]) if case["bare"] else ends
        state["max"] = None if case["bare"] else max(lens)
    if case["train"]:
        state["do"] = rows()
        state["drem"] = torch.randn(lead + (heads, tokens), generator=g, device="cuda", dtype=dtype)
        for x in (q, k, v):
            x.requires_grad_()
    return state


def _forward(state):
    case, q, k, v = state["case"], state["q"], state["k"], state["v"]
    if case["layout"] == "batched":
        return sb_attn(q, k, v, attend_current=case["current"], fuse_remainder=case["fuse"])
    return sb_attn_varlen(q, k, v, state["cu"], state["max"], zero_start=case["bare"], attend_current=case["current"],
                          fuse_remainder=case["fuse"])


def run(state):
    if not state["case"]["train"]:
        with torch.no_grad():
            o, rem = _forward(state)
        return {"o": o, "rem": rem}
    o, rem = _forward(state)
    dq, dk, dv = torch.autograd.grad([o, rem], [state["q"], state["k"], state["v"]], [state["do"], state["drem"]])
    return {"o": o, "rem": rem, "dq": dq, "dk": dk, "dv": dv}


def work(case):
    """Every visible (query, key) pair costs 4 D flops forward (Q K^T, P V) and 10 D backward (Q K^T again, dO V^T, dQ, dK, dV);
    q, k, v (and do, drem) are read once, o, rem (and dq, dk, dv) written once."""
    batch, tokens, lens = _sizes(case)
    pairs = sum(n * (n + 1) // 2 if case["current"] else n * (n - 1) // 2 for n in lens)
    matrices, vectors = (8, 2) if case["train"] else (4, 1)
    return {"bytes": BYTES[case["dtype"]] * batch * case["heads"] * tokens * (matrices * case["dim"] + vectors),
            "flops": (14 if case["train"] else 4) * case["dim"] * pairs * case["heads"]}


def tolerance(case):
    """The matrices' operands (weights, score gradients) and results have 8 significant bits in bf16 and 11 in f16, sums are float32."""
    return {"rel": {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5}[case["dtype"]]}
