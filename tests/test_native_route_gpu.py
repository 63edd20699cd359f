"""The native eager route (csrc/dm_torch.cpp) against the Python route it stands in for: the same bits over layouts, head dims,
modes, arms and a bounded workspace, although its backward may take other kernels (tests/test_small_grids_gpu.py)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(fn, leaves, do):
    o = fn(leaves)
    return (o.detach(),) + torch.autograd.grad(o, leaves, do)


@pytest.mark.parametrize("B,N,H,Hk,D,causal,mode,numerics,layout,cap_mb", [
    (1, 256, 2, 2, 128, True, "matched", "sm100-mx", "dense", None),
    (3, 512, 6, 2, 128, True, "matched", "sm100-mx-ds32", "packed", None),
    (2, 256, 3, 1, 128, False, "stale", "sm100-mx", "bhnd", None),
    (2, 512, 4, 2, 128, True, "matched", "sm100-mx-nonorm", "odd_strides", "1"),     # split over ops.bwd_fp8; rows that need a copy
    (1, 384, 2, 1, 256, True, "matched", "sm100-mx-d256", "bhnd", None),
])
def test_native_route_equals_python_route(B, N, H, Hk, D, causal, mode, numerics, layout, cap_mb, oracle, monkeypatch):
    from delta_matching_b200 import _lib, dm_attn_func, dm_attn_func_bhnd
    q, k, v, do = oracle.make_inputs(B, N, H, Hk, D, seed=61, device="cuda")
    if layout == "packed":
        q, k, v = torch.cat((q, k, v), dim=2).split([H, Hk, Hk], dim=2)
    elif layout == "bhnd":
        q, k, v = (t.transpose(1, 2).contiguous() for t in (q, k, v))
    elif layout == "odd_strides":
        wide = torch.zeros(B, N, H, D + 4, device="cuda", dtype=torch.bfloat16)
        wide[..., :D] = q
        q, do = wide[..., :D], do.sum().expand(B, N, H, D)
    if cap_mb is not None:
        monkeypatch.setenv("DM_BWD_WORKSPACE_MB", cap_mb)
    leaves = [t.detach().requires_grad_() for t in (q, k, v)]
    if layout == "bhnd":
        call = lambda x: dm_attn_func_bhnd(*x, causal=causal, delta_mode=mode, numerics=numerics)
    else:
        call = lambda x: dm_attn_func(*x, causal=causal, mode=mode, numerics=numerics)
    got = _step(call, leaves, do)
    with torch.no_grad():
        o = call(leaves)
    monkeypatch.setattr(_lib, "_NATIVE", _lib._decline)
    want = _step(call, leaves, do)
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert a.shape == b.shape and a.stride() == b.stride() and torch.equal(a, b)
    assert torch.equal(o, want[0])


def test_second_derivative_is_refused(oracle):
    from delta_matching_b200 import dm_attn_func
    q, k, v, do = oracle.make_inputs(1, 256, 2, 2, 128, seed=62, device="cuda")
    leaves = [t.requires_grad_() for t in (q, k, v)]
    o = dm_attn_func(*leaves, causal=True)
    (dq,) = torch.autograd.grad(o, leaves[:1], do.requires_grad_(), create_graph=True)
    with pytest.raises(RuntimeError, match="once_differentiable"):
        dq.sum().backward()


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("mode", ["matched", "stale"])
def test_jit_trace_records_the_call(mode, grad, oracle):
    """A traced function gives the eager result on inputs other than those it was traced with."""
    from delta_matching_b200 import dm_attn_func
    f = lambda q, k, v: 2.0 * dm_attn_func(q, k, v, causal=True, mode=mode)
    one, two = (oracle.make_inputs(1, 256, 2, 2, 128, seed=s, device="cuda") for s in (63, 64))
    traced = torch.jit.trace(f, [t.requires_grad_(grad) for t in one[:3]], check_trace=False)
    got, want = ([t.detach().requires_grad_(grad) for t in two[:3]] for _ in range(2))
    a, b = traced(*got), f(*want)
    assert torch.equal(a, b)
    if grad:
        for x, y in zip(torch.autograd.grad(a, got, two[3]), torch.autograd.grad(b, want, two[3])):
            assert torch.equal(x, y)
