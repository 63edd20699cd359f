"""dK and dV of a grid that fills the SMs (persistent CTAs, items of one after the other) against the same units in grids that do not
(a CTA per key tile and role): the bits of a unit must not depend on how many units the call has."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,Hk,causal,ds32", [
    (40, 256, 1, 1, True, False),       # an item per CTA: of two tiles, or of one
    (74, 256, 1, 1, True, True),        # exactly an item per SM
    (75, 256, 2, 1, False, False),      # two CTAs take a second item
    (40, 512, 2, 2, True, False),       # items of one to four tiles, several per CTA
    (20, 512, 3, 1, True, True),
    (9, 1024, 5, 1, False, True),       # the stage ring wraps inside an item and across items
    (3, 1792, 15, 5, True, False),
])
def test_units_have_the_bits_of_a_small_grid(B, N, H, Hk, causal, ds32, oracle):
    from delta_matching_b200 import ops
    q, k, v, do = (t.transpose(1, 2) for t in oracle.make_inputs(B, N, H, Hk, 128, seed=75, device="cuda"))
    q8, qs, k8, ks, v8, vs, _ = ops.quant_qkv(q, k, v)
    do8, dos, _ = ops.quant_do(do)
    _, lse = ops.fwd_fp8(q8, k8, v8, qs, ks, vs, causal)
    delta = ops.delta_fp8(q8, k8, v8, do8, qs, ks, vs, dos, lse, causal)
    args = (q8, k8, v8, do8, qs, ks, vs, dos, lse, delta)
    whole = ops.bwd_fp8(*args, causal, ds32=ds32)
    bare = ops.bwd_fp8(*args, causal, identity=True, ds32=ds32)      # no workspace: the dS tiles stay where they are
    for b in (0, B // 2, B - 1):
        part = ops.bwd_fp8(*(t[b:b + 1] for t in args), causal, ds32=ds32)
        for nm, x, y in zip(("dQ", "dK", "dV"), whole, part):
            assert torch.equal(x[b:b + 1], y), nm
    for nm, x, y in zip(("dK", "dV"), whole[1:], bare[1:]):
        assert torch.equal(x, y), nm
    ops.check_status()
