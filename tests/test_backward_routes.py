"""The line between the two backwards of dm_attn_bwd: which side of it a call is on, by the workspace that it asks for (both tile sets or
the dS tiles alone; B200's 148 SMs, which the library also assumes without a GPU), and the same bits on either side."""
import pytest
import torch

# head_dim 128, bidirectional: tile-parallel up to 68 key tiles (B Hk N / 128); causal: from a chain of 2.25 tiles per SM's share on
CALLS = [(1, 2816, 12, 3, False, True), (17, 512, 4, 1, False, True), (1, 4352, 2, 2, False, True), (1, 1280, 28, 7, False, False),
         (35, 256, 4, 1, False, False), (2, 2304, 2, 2, False, False), (37, 256, 4, 1, False, False),
         (1, 16384, 2, 1, True, True), (1, 8192, 8, 2, True, True), (1, 4096, 16, 4, True, False), (4, 1024, 16, 4, True, False)]


def _tile_parallel(B, N, H, Hk, causal):
    from delta_matching_b200 import _lib, ops
    need, ds_only = _lib.lib().dm_attn_bwd_workspace_bytes(B, N, H, Hk, 128, int(causal)), ops.bwd_workspace_bytes(B, N, H, 128)
    tiles = B * H * (N // 128) ** 2
    assert ds_only == tiles * (16384 + 16) and need in (ds_only, tiles * (2 * 16384 + 16 + 512))
    return need != ds_only


@pytest.mark.parametrize("B,N,H,Hk,causal,tile_parallel", CALLS)
def test_side_of_the_line(B, N, H, Hk, causal, tile_parallel):
    assert _tile_parallel(B, N, H, Hk, causal) == tile_parallel


@pytest.mark.gpu
@pytest.mark.parametrize("B,N,H,Hk,causal,tile_parallel", [c for c in CALLS if not c[4]])
@pytest.mark.parametrize("numerics", ["sm100-mx", "sm100-mx-ds32"])
def test_bits_at_the_line(B, N, H, Hk, causal, tile_parallel, numerics, oracle):
    """dm_attn_func takes the form named above, the op layer the key-stationary one."""
    from .helpers import run_api, run_ops
    q, k, v, do = oracle.make_inputs(B, N, H, Hk, 128, seed=77, device="cuda")
    got = run_api(q, k, v, do, causal, "stale", numerics)
    want = run_ops(q, k, v, do, causal, "stale", numerics=numerics)
    for nm in ("dQ", "dK", "dV"):
        assert torch.equal(got[nm], want[nm]), nm
