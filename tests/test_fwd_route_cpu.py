"""Which of the two forwards of head_dim 128 a shape takes (host only: B200's 148 SMs, which the library also assumes without a GPU)."""
import pytest

# (B, N, H, Hk, D, causal), whether dm_fwd takes the three teams
CALLS = [((1, 1024, 8, 2, 128, True), True), ((1, 4096, 9, 9, 128, True), True), ((1, 8192, 6, 1, 128, True), True),
         ((8, 2048, 16, 16, 128, False), True), ((4, 4096, 32, 8, 128, True), False), ((1, 2048, 6, 2, 256, True), False)]


def _route(shape, unordered=0):
    from delta_matching_b200 import _lib
    return _lib.lib().dm_dbg_fwd_kernel(*(int(x) for x in shape), unordered)


@pytest.mark.parametrize("shape,teams", CALLS)
def test_route(shape, teams):
    assert _route(shape) == int(teams)


@pytest.mark.parametrize("shape", [c[0] for c in CALLS])
def test_the_form_without_the_ordering_wait_never_takes_the_teams(shape):
    """Two threads issue the teams' S and PV chains: there is no issue order between them to rely on."""
    assert _route(shape, unordered=1) == 0


def test_route_of_a_refused_shape():
    assert _route((1, 100, 1, 1, 128, True)) < 0


@pytest.mark.parametrize("D,kernel", [(256, 1), (128, 2), (128, -1)])
def test_no_such_kernel(D, kernel):
    from delta_matching_b200 import _lib
    rc = _lib.lib().dm_dbg_fwd_forced(None, None, None, None, None, None, 1, 256, 1, 1, D, 1, None, 0, 0, 0, None, None, None, kernel)
    assert rc < 0 and "no forward kernel" in _lib.last_error()


# Bidirectional chains of one and three key tiles, whose few rounds of items measured slower in the teams
@pytest.mark.parametrize("N,heads,teams", [(128, 16, False), (128, 148, False), (128, 441, False), (128, 1033, False), (128, 1329, True), (384, 49, True),
                                           (384, 147, True), (384, 207, False), (384, 246, False), (384, 443, True), (256, 71, True), (512, 184, True)])
def test_route_of_short_bidirectional_chains(N, heads, teams):
    assert _route((1, N, heads, heads, 128, False)) == int(teams)


# Causal calls of short chains close to two items per SM: six key tiles measured slower in the teams there, seven did not
@pytest.mark.parametrize("N,heads,teams", [(768, 36, True), (768, 42, True), (768, 48, False), (768, 49, False), (896, 40, True), (1024, 36, True)])
def test_route_of_short_causal_chains(N, heads, teams):
    assert _route((1, N, heads, heads, 128, True)) == int(teams)
