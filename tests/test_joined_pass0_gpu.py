"""Pass 0 that quantises its own dO tiles (as many items as SMs at most) against the producer and pass 0 as two launches."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,H,Hk,D,numerics", [
    (1, 256, 1, 1, 128, "sm100-mx"),
    (1, 256, 2, 2, 128, "sm100-mx-nonorm"),
    (2, 1024, 8, 2, 128, "sm100-mx"),         # 128 items of up to 8 key tiles
    (1, 18944, 1, 1, 128, "sm100-mx"),        # exactly an item per SM, chains past every ring
    (1, 19200, 1, 1, 128, "sm100-mx"),        # one item more: two launches
    (1, 128, 3, 1, 256, "sm100-mx"),
    (1, 1920, 6, 2, 256, "sm100-mx-d256-ds32"),
])
@pytest.mark.parametrize("strided", [False, True])
def test_same_bits_as_two_launches(B, N, H, Hk, D, numerics, strided, oracle):
    """dm_attn_func quantises dO in pass 0 where it can, the op layer never."""
    from .helpers import run_api, run_ops
    q, k, v, do = oracle.make_inputs(B, N, H, Hk, D, seed=76, device="cuda")
    if strided:                               # dO as a slice of a wider buffer, with rows that differ in size by many binades
        do = do * torch.logspace(-6, 6, N, base=2.0, device="cuda").view(1, N, 1, 1).to(do.dtype)
        wide = torch.zeros(B, N, H, 2 * D, device="cuda", dtype=do.dtype)
        wide[..., D:] = do
        do = wide[..., D:]
    got = run_api(q, k, v, do, True, "matched", numerics)
    want = run_ops(q, k, v, do, True, "matched", numerics=numerics)
    for nm in ("dQ", "dK", "dV"):
        assert torch.equal(got[nm], want[nm]), nm


def test_first_cuda_call_of_the_autograd_thread():
    """The tensor maps of the backward are then encoded before anything else has made a context current on that thread."""
    code = ("import torch, delta_matching_b200 as dm\n"
            "q, k, v = (torch.randn(1, 256, 2, 128, device='cuda', dtype=torch.bfloat16, requires_grad=True) for _ in range(3))\n"
            "o = dm.dm_attn_func(q, k, v, causal=True)\n"
            "g = torch.autograd.grad(o, (q, k, v), torch.randn_like(o))\n"
            "torch.cuda.synchronize(); assert all(bool(t.isfinite().all()) for t in g)\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
