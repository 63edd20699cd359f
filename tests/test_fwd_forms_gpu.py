"""The two forwards of head_dim 128: one CTA per SM with three teams of softmax warps, and two CTAs per SM.  Which one a call takes depends
on its size only, and what a query tile computes must not: each kernel by name on the same codes, and on single units of them (one work item
per CTA there, several in the whole call)."""
import pytest
import torch

from .helpers import fwd_forced

pytestmark = pytest.mark.gpu


def _codes(oracle, N, rep, items_per_sm, scale):
    from delta_matching_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    units = max(3, round(items_per_sm * sms / (N // 128 * rep)))
    q, k, v, _ = oracle.make_inputs(units, N, rep, 1, 128, seed=74, device="cuda", qk_scale=scale)
    q8, qs, k8, ks, v8, vs = ops.quant_qkv(*(t.transpose(1, 2) for t in (q, k, v)))[:6]
    return q8, k8, v8, qs, ks, vs


@pytest.mark.parametrize("N,rep,causal,scale,items_per_sm", [
    (128, 1, False, 1.0, 7.3),    # a single key tile: every item is another team's
    (128, 2, True, 3.0, 2.0),
    (512, 1, True, 1.0, 6.0),     # items of one to four key tiles: teams without a tile of their item
    (512, 2, False, 12.0, 6.0),
    (1024, 1, True, 12.0, 6.0),   # the running maximum moves by more than 32 binades between key tiles: O is rescaled by another team
    (1024, 1, True, 12.0, 1.7),   # some CTAs walk two items, others one
    (768, 3, False, 1.0, 6.0),    # six tiles: two per team
    (1280, 1, True, 12.0, 6.0),   # ten tiles: no multiple of the teams or of the stages
    (1280, 1, True, 1.0, 1.9),
    (1792, 3, True, 3.0, 6.0),
    (2048, 1, True, 3.0, 2.4),    # three items on some CTAs
    (2048, 1, False, 3.0, 6.0),   # O of an item leaves under the next one
    (4096, 2, True, 12.0, 6.0),
    (8192, 2, True, 12.0, 4.0),
])
def test_a_unit_has_the_same_bits_in_both_forwards(N, rep, causal, scale, items_per_sm, oracle):
    from delta_matching_b200 import ops
    codes = _codes(oracle, N, rep, items_per_sm, scale)
    pairs, teams, by_rule = fwd_forced(codes, causal, 0), fwd_forced(codes, causal, 1), ops.fwd_fp8(*codes, causal)
    assert torch.isfinite(pairs[0].float()).all() and torch.isfinite(pairs[1]).all()
    for got in (teams, by_rule):
        assert torch.equal(got[0], pairs[0]) and torch.equal(got[1], pairs[1])
    units = codes[0].shape[0]
    for u in (0, units // 2, units - 1):
        one = [t[u:u + 1].contiguous() for t in codes]
        for kernel in (0, 1):
            o1, lse1 = fwd_forced(one, causal, kernel)
            assert torch.equal(o1, pairs[0][u:u + 1]) and torch.equal(lse1, pairs[1][u:u + 1]), (u, kernel)
        o1, lse1 = ops.fwd_fp8(*one, causal, unordered=True)
        assert torch.equal(o1, pairs[0][u:u + 1]) and torch.equal(lse1, pairs[1][u:u + 1]), u
    ops.check_status("cuda")


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("layout", ["head-major", "padded rows"])
def test_strided_output(layout, kernel, oracle):
    """O by the strides that dm_fwd takes, at several work items per CTA; nothing beside its elements is written."""
    N, rep = 640, 3
    codes = _codes(oracle, N, rep, 6.0, 1.0)
    B = codes[0].shape[0]
    want = fwd_forced(codes, True, 0)
    if layout == "head-major":
        buf = torch.full((B, rep, N + 1, 128), 7.0, device="cuda", dtype=torch.bfloat16)
        view, rest = buf[:, :, :N].transpose(1, 2), (buf[:, :, N:],)
    else:
        buf = torch.full((B, N, rep + 1, 136), 7.0, device="cuda", dtype=torch.bfloat16)
        view, rest = buf[:, :, :rep, :128], (buf[:, :, rep], buf[..., 128:])
    o, lse = fwd_forced(codes, True, kernel, o=view)
    assert torch.equal(o, want[0]) and torch.equal(lse, want[1])
    for r in rest:
        assert (r == 7.0).all()


@pytest.mark.parametrize("B,N,H,Hk,causal,scale", [(4, 4096, 32, 8, True, 1.0), (8, 2048, 16, 16, False, 30.0)])
def test_the_ordering_wait_changes_no_bit_of_the_pairs(B, N, H, Hk, causal, scale, oracle):
    """The kernel whose one thread issues S and PV, with its wait between the two and without: dm_fwd takes the teams for the second shape,
    so the ordered side is named."""
    from delta_matching_b200 import ops
    q, k, v, _ = oracle.make_inputs(B, N, H, Hk, 128, seed=5, device="cuda", qk_scale=scale)
    q8, qs, k8, ks, v8, vs = ops.quant_qkv(*(t.transpose(1, 2) for t in (q, k, v)))[:6]
    codes = (q8, k8, v8, qs, ks, vs)
    want = fwd_forced(codes, causal, 0)
    for i in range(20):
        ordered, unordered = fwd_forced(codes, causal, 0), ops.fwd_fp8(*codes, causal, unordered=True)
        for name, got in (("ordered", ordered), ("unordered", unordered)):
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (name, i)
    ops.check_status("cuda")
