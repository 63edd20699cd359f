"""The two forwards of head_dim 128: one CTA per SM with three teams of softmax warps, and two CTAs per SM.  Which one a call takes depends
on its size only, and what a query tile computes must not: the units of a call with several work items per SM (short sequences: the pairs of CTAs),
against the same units in a call of their own, which the teams take."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,rep,causal,scale", [
    (512, 1, True, 1.0),          # items of one to four key tiles: teams without a tile of their item
    (512, 2, False, 12.0),
    (1024, 1, True, 12.0),        # the running maximum moves by more than 32 binades between key tiles: O is rescaled by another team
    (768, 3, False, 1.0),         # one tile per team
    (1280, 1, True, 12.0),        # ten tiles: no multiple of the teams or of the stages
    (1792, 3, True, 3.0),
    (2048, 1, False, 3.0),        # six items per CTA, which the teams take in the large call too: O of an item leaves under the next one
    (4096, 2, True, 12.0),
])
def test_a_unit_has_the_same_bits_in_both_forwards(N, rep, causal, scale, oracle):
    from delta_matching_b200 import ops
    n_t = N // 128
    units = -(-6 * torch.cuda.get_device_properties(0).multi_processor_count // (n_t * rep))
    q, k, v, _ = oracle.make_inputs(units, N, rep, 1, 128, seed=74, device="cuda", qk_scale=scale)
    q8, qs, k8, ks, v8, vs = ops.quant_qkv(*(t.transpose(1, 2) for t in (q, k, v)))[:6]
    o, lse = ops.fwd_fp8(q8, k8, v8, qs, ks, vs, causal)
    for u in (0, units // 2, units - 1):
        one = [t[u:u + 1].contiguous() for t in (q8, k8, v8, qs, ks, vs)]
        for unordered in (False, True):
            o1, lse1 = ops.fwd_fp8(*one, causal, unordered=unordered)
            assert torch.equal(o1, o[u:u + 1]) and torch.equal(lse1, lse[u:u + 1]), (u, unordered)
    ops.check_status("cuda")
