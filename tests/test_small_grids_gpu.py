"""The variants that small problems take, against the forms that large ones take: the producers of a short sequence in one
launch, dK and dV as two roles, the tile-parallel backward.  What a (batch, head) unit computes must not depend on
how many units the call has, so the bits of a small call are those of the same units inside a large one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,Hk,D", [(1, 256, 2, 1, 128), (2, 512, 3, 3, 128), (1, 128, 2, 2, 256), (3, 256, 2, 1, 256),
                                         (2, 768, 4, 2, 128), (1, 2304, 2, 1, 128), (1, 384, 2, 2, 256), (1, 4096, 1, 1, 256)])
def test_joined_producers_equal_the_separate_ones(B, N, H, Hk, D, oracle):
    from delta_matching_b200 import ops
    q, k, v, _ = (t.transpose(1, 2) for t in oracle.make_inputs(B, N, H, Hk, D, seed=71, device="cuda"))
    k = k + 0.5
    q8, qs, k8, ks, v8, vs, km = ops.quant_qkv(q, k, v)
    mean = ops.kmean(k)
    assert torch.equal(km, mean)
    for (codes, scales), (c, s) in (((q8, qs), ops.quant_rows(q, D ** -0.5)), ((k8, ks), ops.quant_rows(k, 1.0, mean)), ((v8, vs), ops.quant_rows(v))):
        assert torch.equal(codes.view(torch.uint8), c.view(torch.uint8)) and torch.equal(scales, s)


@pytest.mark.parametrize("B,N,H,Hk,D,causal,mode,numerics", [
    (1, 256, 2, 2, 128, True, "matched", "sm100-mx"),              # fewer tiles than SMs
    (1, 1024, 8, 1, 128, True, "matched", "sm100-mx"),             # two or three tiles per CTA, key tiles change inside one
    (2, 1536, 6, 2, 128, False, "stale", "sm100-mx-ds32"),
    (1, 4096, 4, 1, 128, True, "stale", "sm100-mx"),               # many tiles per CTA: every ring wraps
    (1, 128, 3, 1, 256, True, "matched", "sm100-mx"),
    (1, 1920, 6, 2, 256, False, "stale", "sm100-mx"),
    (1, 1664, 4, 1, 256, True, "matched", "sm100-mx-d256-ds32"),
])
def test_tile_parallel_backward_equals_the_key_stationary_one(B, N, H, Hk, D, causal, mode, numerics, oracle):
    """dm_attn_func takes the tile-parallel backward for these shapes, the op layer always the key-stationary one."""
    from delta_matching_b200 import _lib, ops
    from .helpers import run_api, run_ops
    assert _lib.lib().dm_attn_bwd_workspace_bytes(B, N, H, Hk, D, int(causal)) > ops.bwd_workspace_bytes(B, N, H, D)
    q, k, v, do = oracle.make_inputs(B, N, H, Hk, D, seed=73, device="cuda")
    got = run_api(q, k, v, do, causal, mode, numerics)
    want = run_ops(q, k, v, do, causal, mode, numerics=numerics)
    for nm in ("dQ", "dK", "dV"):
        assert torch.equal(got[nm], want[nm]), nm


@pytest.mark.parametrize("N,rep,D,causal,mode,scale", [(256, 1, 128, True, "matched", 1.0), (1280, 3, 128, True, "matched", 4.0), (768, 2, 128, False, "stale", 12.0),
                                                       (384, 1, 256, True, "matched", 1.0), (640, 2, 256, False, "stale", 6.0)])
def test_a_unit_has_the_same_bits_in_a_small_and_a_large_call(N, rep, D, causal, mode, scale, oracle):
    import delta_matching_b200 as dm
    units = -(-160 // (N // 128))                        # more work items than SMs
    q, k, v, do = oracle.make_inputs(units, N, rep, 1, D, seed=72, device="cuda", qk_scale=scale)

    def step(b0, b1):
        leaves = [t[b0:b1].detach().requires_grad_() for t in (q, k, v)]
        o = dm.dm_attn_func(*leaves, causal=causal, mode=mode)
        return (o.detach(),) + torch.autograd.grad(o, leaves, do[b0:b1])

    whole = step(0, units)
    for u in (0, units - 1):
        for a, b in zip(step(u, u + 1), whole):
            assert torch.equal(a, b[u:u + 1])


@pytest.mark.parametrize("B,N,H,Hk,causal,mode,numerics", [
    (5, 8192, 8, 8, True, "matched", "sm100-mx"),            # ranges of three and two batches
    (1, 16384, 8, 4, True, "stale", "sm100-mx-d256-ds32"),   # two ranges of two kv groups
    (3, 16384, 3, 3, False, "stale", "sm100-mx"),            # two batches, then one
    (1, 16384, 9, 9, True, "matched", "sm100-mx"),           # kv groups in ranges of five and four
])
def test_ranges_of_the_wide_backward_equal_the_op_layer(B, N, H, Hk, causal, mode, numerics, oracle):
    """Head_dim 256 calls whose two tile sets exceed one range: dm_attn_func goes range by range through the P^T form, the op layer
    through the key-stationary kernel."""
    from delta_matching_b200 import _lib, ops
    from .helpers import run_api, run_ops
    per_head = (N // 128) ** 2 * (2 * 16384 + 528)
    ws = _lib.lib().dm_attn_bwd_workspace_bytes(B, N, H, Hk, 256, int(causal))
    assert ops.bwd_workspace_bytes(1, N, 1, 256) < ws < B * H * per_head and ws % per_head == 0
    q, k, v, do = oracle.make_inputs(B, N, H, Hk, 256, seed=74, device="cuda")
    got = run_api(q, k, v, do, causal, mode, numerics)
    want = run_ops(q, k, v, do, causal, mode, numerics=numerics)
    for nm in ("dQ", "dK", "dV"):
        assert torch.equal(got[nm], want[nm]), nm
