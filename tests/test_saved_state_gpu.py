"""What the autograd node of the eager route (csrc/dm_torch.cpp) keeps for its backward: a second pass over a retained graph, and
saved_tensors_hooks, which may bring the saved tensors back from elsewhere and in another layout."""
import pytest
import torch
from torch.autograd.graph import save_on_cpu, saved_tensors_hooks

pytestmark = pytest.mark.gpu

CASES = [(1, 512, 4, 2, 128, "matched"), (2, 256, 3, 1, 128, "stale"), (1, 384, 2, 2, 256, "stale")]


def _setup(oracle, B, N, H, Hk, D, mode, seed):
    from delta_matching_b200 import dm_attn_func
    q, k, v, do = oracle.make_inputs(B, N, H, Hk, D, seed=seed, device="cuda")
    leaves = [t.requires_grad_() for t in (q, k, v)]
    call = lambda: dm_attn_func(*leaves, causal=True, mode=mode)
    return leaves, do, call


@pytest.mark.parametrize("B,N,H,Hk,D,mode", CASES)
def test_second_backward_over_a_retained_graph(B, N, H, Hk, D, mode, oracle):
    leaves, do, call = _setup(oracle, B, N, H, Hk, D, mode, 91)
    o = call()
    first = torch.autograd.grad(o, leaves, do, retain_graph=True)
    other = torch.autograd.grad(o, leaves, -2 * do, retain_graph=True)
    again = torch.autograd.grad(o, leaves, do)
    for a, b, c in zip(first, again, other):
        assert torch.equal(a, b) and torch.equal(c, -2 * a)          # powers of two scale the codes' scales only
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o, leaves, do)


def _other_layout(t):
    """The same values over a storage in another order."""
    if t.dim() == 4:
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    return torch.stack((t, t), dim=1)[:, 0]


@pytest.mark.parametrize("hooks", [lambda: save_on_cpu(pin_memory=True), lambda: saved_tensors_hooks(lambda t: t.clone(), lambda t: t),
                                   lambda: saved_tensors_hooks(_other_layout, lambda t: t)], ids=["cpu", "clone", "layout"])
@pytest.mark.parametrize("B,N,H,Hk,D,mode", CASES)
def test_saved_tensors_hooks(B, N, H, Hk, D, mode, hooks, oracle):
    leaves, do, call = _setup(oracle, B, N, H, Hk, D, mode, 92)
    want = torch.autograd.grad(call(), leaves, do)
    with hooks():
        o = call()
    got = torch.autograd.grad(o, leaves, do)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("change", [lambda t: t[1:] if t.dim() == 1 else t, lambda t: t.to(torch.int16) if t.dim() == 1 else t,
                                    lambda t: t.cpu(), lambda t: t.float() if t.dim() == 4 else t, lambda t: t[:, :, :1] if t.dim() == 4 else t],
                         ids=["fewer bytes", "wider codes", "cpu", "fp32 O", "one head"])
def test_saved_tensors_that_come_back_changed_are_refused(change, oracle):
    leaves, do, call = _setup(oracle, 1, 256, 2, 2, 128, "stale", 93)
    with saved_tensors_hooks(lambda t: t, change):
        o = call()
    with pytest.raises(RuntimeError, match="must come back from saved-tensor hooks"):
        torch.autograd.grad(o, leaves, do)
