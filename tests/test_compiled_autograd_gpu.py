"""Backward passes of the eager route under compiled autograd: the node in csrc/dm_torch.cpp serves it as a Python
autograd.Function does, as one opaque call of the recorded graph."""
import pytest
import torch
import torch._dynamo

pytestmark = pytest.mark.gpu


def _leaves(tensors):
    return [t.detach().requires_grad_() for t in tensors]


@pytest.mark.parametrize("B,N,H,Hk,D,mode,numerics,layout", [
    (1, 256, 2, 2, 128, "matched", "sm100-mx", "dense"),
    (2, 512, 4, 2, 128, "stale", "sm100-mx", "dense"),
    (1, 256, 4, 1, 128, "matched", "sm100-mx-ds32", "bhnd"),
    (1, 384, 2, 1, 256, "stale", "sm100-mx", "bhnd"),
])
@pytest.mark.parametrize("compiler", ["graph", "eager"])
def test_backward_under_compiled_autograd(B, N, H, Hk, D, mode, numerics, layout, compiler, oracle):
    """compiler: the recorded graph run as it is, or through torch.compile.  Two passes per call, so that the second one runs from the cached graph on tensors of its own."""
    from torch._dynamo import compiled_autograd
    from delta_matching_b200 import dm_attn_func, dm_attn_func_bhnd
    if layout == "bhnd":
        call = lambda x: dm_attn_func_bhnd(*x, causal=True, delta_mode=mode, numerics=numerics)
    else:
        call = lambda x: dm_attn_func(*x, causal=True, mode=mode, numerics=numerics)
    torch._dynamo.reset()
    compiler_fn = (lambda gm: gm) if compiler == "graph" else (lambda gm: torch.compile(gm, backend="eager"))
    for seed in (81, 82):
        q, k, v, do = oracle.make_inputs(B, N, H, Hk, D, seed=seed, device="cuda")
        if layout == "bhnd":
            q, k, v = (t.transpose(1, 2).contiguous() for t in (q, k, v))
        want, got = _leaves((q, k, v)), _leaves((q, k, v))
        (call(want) * 2.0).backward(do)
        loss = call(got) * 2.0
        with compiled_autograd._enable(compiler_fn):
            loss.backward(do)
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a.grad, b.grad)
