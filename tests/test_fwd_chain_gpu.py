"""The forward in three teams inside a run of kernels: what is launched behind it must see all of O and LSE, and must not run slower for
having started on SMs that the teams have just left."""
import statistics

import pytest
import torch

from .helpers import fwd_forced

pytestmark = pytest.mark.gpu


def _inputs(heads, N, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(1, heads, N, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(3)]


def _codes(q, k, v):
    from delta_matching_b200 import ops
    q8, qs, k8, ks, v8, vs = ops.quant_qkv(q, k, v)[:6]
    return q8, k8, v8, qs, ks, vs


@pytest.mark.parametrize("heads,N", [(3, 256), (37, 512), (301, 256), (75, 1024)])     # part of the SMs; one item each; several
def test_the_next_kernel_reads_a_complete_output(heads, N):
    from delta_matching_b200 import ops
    runs = [_inputs(heads, N, seed) for seed in range(4)]
    want = []
    for x in runs:
        codes = _codes(*x)
        torch.cuda.synchronize()
        o, lse = fwd_forced(codes, True, 1)
        torch.cuda.synchronize()
        want.append((o, lse, *ops.quant_do(x[0], o.permute(0, 2, 1, 3))))
        torch.cuda.synchronize()
    got = []
    for x in runs:
        o, lse = fwd_forced(_codes(*x), True, 1)
        got.append((o, lse, *ops.quant_do(x[0], o.permute(0, 2, 1, 3))))
    for w, g in zip(want, got):
        for a, b in zip(w, g):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))


def test_the_producers_keep_their_pace_behind_the_teams():
    """Time of (producers, forward) in a run, less that of forwards alone, against the producers alone.  Equal but for the boundary of two kernels; a fifth
    more where the producers start on SMs that still have the teams' division of L1 and shared memory.  Half way between is the limit."""
    from delta_matching_b200 import ops
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = _inputs(41 * sms, 128, 7)
    codes = _codes(*x)
    calls = {"both": lambda: fwd_forced(_codes(*x), False, 1), "forward": lambda: fwd_forced(codes, False, 1), "producers": lambda: ops.quant_qkv(*x)}
    times = {name: [] for name in calls}
    for turn in range(7):
        for name, call in calls.items():
            call()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            a.record()
            for _ in range(40):
                call()
            b.record()
            torch.cuda.synchronize()
            times[name].append(a.elapsed_time(b) / 40)
    both, forward, producers = (statistics.median(times[n]) for n in ("both", "forward", "producers"))
    assert both - forward < 1.1 * producers, (both, forward, producers)
