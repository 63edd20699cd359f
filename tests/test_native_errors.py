"""Errors raised in the native eager route (csrc/dm_torch.cpp) reach Python as exceptions, from the forward and from the autograd
engine's threads."""
import ctypes
import os

import pytest
import torch


def test_native_module_shares_the_cxx_runtime():
    """An exception thrown by one copy of the C++ runtime and caught by torch's ends the process."""
    import __graft_entry__ as entry
    import delta_matching_b200
    entry.build()
    native = ctypes.CDLL(os.path.join(os.path.dirname(delta_matching_b200.__file__), "_dm_native.so"))
    address = lambda lib: ctypes.cast(getattr(lib, "__cxa_throw"), ctypes.c_void_p).value
    assert address(native) == address(ctypes.CDLL("libstdc++.so.6"))


def _leaves(oracle, seed):
    q, k, v, do = oracle.make_inputs(1, 256, 2, 2, 128, seed=seed, device="cuda")
    return [t.requires_grad_() for t in (q, k, v)], do


@pytest.mark.gpu
def test_contiguous_but_misaligned_tensors_are_refused(oracle):
    """A contiguous view 2 bytes off a 16-byte boundary: no copy is made of it, the entry points refuse it."""
    from delta_matching_b200 import dm_attn_func
    leaves, do = _leaves(oracle, 95)
    off = lambda t: torch.cat((t.new_zeros(1), t.detach().flatten()))[1:].view(t.shape)
    for i in range(3):
        with pytest.raises(RuntimeError, match="16-byte aligned"):
            dm_attn_func(*(off(t) if i == j else t for j, t in enumerate(leaves)), causal=True)
    with pytest.raises(RuntimeError, match="16-byte aligned"):
        torch.autograd.grad(dm_attn_func(*leaves, causal=True), leaves, off(do))


@pytest.mark.gpu
def test_reported_status_raises_in_the_backward(oracle):
    """A status that a kernel left behind, set by the host here: the next pass raises it and the one after that runs."""
    from delta_matching_b200 import dm_attn_func, ops
    leaves, do = _leaves(oracle, 96)
    want = torch.autograd.grad(dm_attn_func(*leaves, causal=True), leaves, do)
    o = dm_attn_func(*leaves, causal=True)
    torch.cuda.synchronize()
    ops.status_word("cuda")[0] = 0x13
    with pytest.raises(RuntimeError, match="reported status 19"):
        torch.autograd.grad(o, leaves, do)
    got = torch.autograd.grad(dm_attn_func(*leaves, causal=True), leaves, do)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
