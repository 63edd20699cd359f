"""What this package is timed on: calls of its public attention functions over the range of shapes they are used at.

A case is one attention layer's call: `train` = forward and backward (the gradients of q, k and v for a given dO), `eval` =
forward alone without a graph.  q and dO have shape (B, N, H, D), k and v (B, N, Hk, D), bf16.  `layout`:
    dense   separate contiguous tensors
    packed  q, k and v are slices of one (B, N, H + 2 Hk, D) tensor, as a fused projection leaves them
    bhnd    contiguous (B, H, N, D) tensors through `dm_attn_func_bhnd`
`qk_scale` multiplies q and k (the range of the logits grows with its square); `qk_norm` brings the rows of q and k to unit
RMS, as models that normalise queries and keys do.
"""
import math

import torch

from delta_matching_b200 import dm_attn_func, dm_attn_func_bhnd


def _case(name=None, **kw):
    c = dict(job="train", B=1, N=256, H=2, Hk=2, D=128, causal=True, mode="matched", numerics="sm100-mx", layout="dense",
             qk_scale=1.0, qk_norm=False)
    c.update(kw)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # the smallest calls: unit tests, probes and toy models, where latency and launches are all there is
        _case("tiny train", B=1, N=256, H=2, Hk=2),
        _case("tiny eval", job="eval", B=1, N=256, H=8, Hk=2),
        # a short sequence of a grouped-query model, one at a time
        _case("short train", B=1, N=1024, H=8, Hk=2),
        # ragged sizes: an odd batch, an odd number of heads per group, a sequence that is no power of two, packed projection
        _case("ragged train packed", B=3, N=1792, H=15, Hk=5, layout="packed"),
        # the layer the benchmark is quoted on (8B-class grouped-query layer), training and evaluation
        _case("layer train", B=4, N=4096, H=32, Hk=8),
        _case("layer eval", job="eval", B=4, N=4096, H=32, Hk=8),
        # the same layer at a micro-batch of one sequence, with the classical delta and head-major tensors
        _case("layer train stale B1", B=1, N=4096, H=32, Hk=8, mode="stale", layout="bhnd"),
        # one device's share of that layer when its heads are split over several, with the finer dS blocks
        _case("layer share ds32", B=2, N=4096, H=16, Hk=4, numerics="sm100-mx-ds32"),
        # head_dim 256: the benchmark's configuration, and a small ragged bidirectional call
        _case("wide head train", B=2, N=8192, H=16, Hk=16, D=256),
        _case("wide head ragged", B=1, N=1920, H=6, Hk=2, D=256, causal=False, mode="stale"),
        # a bidirectional encoder with large logits (the benchmark's logit-range sweep)
        _case("encoder train", B=8, N=2048, H=16, Hk=16, causal=False, mode="stale", qk_scale=3.0),
        # long context: one sequence of the sharded configuration, normalised queries and keys
        _case("long context train", B=1, N=32768, H=64, Hk=8, qk_norm=True),
    ]


def _positions(c):
    """(query, key) pairs that the attention of one head looks at."""
    return c["N"] * (c["N"] + 1) / 2 if c["causal"] else float(c["N"]) ** 2


def work(case):
    c = case
    q, kv = c["B"] * c["N"] * c["H"] * c["D"], c["B"] * c["N"] * c["Hk"] * c["D"]
    matmul = 2.0 * c["B"] * c["H"] * _positions(c) * c["D"]
    if c["job"] == "eval":
        return {"bytes": 2.0 * (2 * q + 2 * kv), "flops": 2 * matmul}      # q k v in, o out; Q K^T and P V
    return {"bytes": 2.0 * (4 * q + 4 * kv), "flops": 7 * matmul}          # q k v dO in, o dq dk dv out; and the five of the backward


_MOST = work(listed()[-1])["flops"]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    while True:
        D = 256 if rng.random() < 0.3 else 128
        step = 256 if D == 128 else 128
        N = step * max(1, round(_log_uniform(rng, 256, 32768 if D == 128 else 16384) / step))
        Hk = max(1, round(_log_uniform(rng, 1, 16)))
        rep = rng.choice([1, 1, 2, 3, 4, 4, 5, 7, 8])
        causal = rng.random() < 0.75
        c = _case(job="eval" if rng.random() < 0.25 else "train", B=max(1, round(_log_uniform(rng, 1, 8))), N=N, H=Hk * rep, Hk=Hk,
                  D=D, causal=causal, mode="matched" if causal and rng.random() < 0.75 else "stale",
                  numerics=rng.choice(["sm100-mx"] * 8 + ["sm100-mx-ds32", "sm100-mx-nonorm"]),
                  layout=rng.choice(["dense", "dense", "packed", "bhnd"]),
                  qk_scale=rng.choice([1.0, 1.0, 1.0, 3.0]), qk_norm=rng.random() < 0.2)
        if c["H"] <= 64 and work(c)["flops"] <= _MOST:
            return c


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)

    B, N, H, Hk, D = c["B"], c["N"], c["H"], c["Hk"], c["D"]
    parts = []
    for heads, is_qk in ((H, True), (Hk, True), (Hk, False)):
        x = rand(B, N, heads, D)
        if is_qk and c["qk_norm"]:
            x = x * torch.rsqrt(x.square().mean(-1, keepdim=True))
        parts.append((x * (c["qk_scale"] if is_qk else 1.0)).to(torch.bfloat16))
        del x
    do = rand(B, N, H, D).to(torch.bfloat16)
    if c["layout"] == "packed":
        parts = list(torch.cat(parts, dim=2).split([H, Hk, Hk], dim=2))
    elif c["layout"] == "bhnd":
        parts = [t.transpose(1, 2).contiguous() for t in parts]
    if c["job"] == "train":
        parts = [t.detach().requires_grad_() for t in parts]
    return {"case": dict(c), "qkv": parts, "do": do}


def run(state):
    c, (q, k, v) = state["case"], state["qkv"]
    if c["layout"] == "bhnd":
        call = lambda: dm_attn_func_bhnd(q, k, v, causal=c["causal"], delta_mode=c["mode"], numerics=c["numerics"])
    else:
        call = lambda: dm_attn_func(q, k, v, causal=c["causal"], mode=c["mode"], numerics=c["numerics"])
    if c["job"] == "eval":
        with torch.no_grad():
            return {"o": call()}
    o = call()
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), state["do"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv}


def tolerance(case):
    # Outputs are bf16 (2^-9 each) of sums over e4m3 codes of P and dS: an exponential that is one unit in the last place away
    # turns a code at a tie into its neighbour (an eighth of that term), which shows most where a row has few keys or one large
    # logit.
    return {"rel": 1e-2, "max": 0.4} if case["qk_scale"] > 1.0 else {"rel": 5e-3, "max": 0.25}
