"""The C-ABI library loads and exports every entry point include/dm_b200.h declares (no GPU needed: nothing is
launched), and the ctypes prototypes cover exactly the declared functions."""
import os
import re

import pytest

from .conftest import ROOT


def _declared():
    text = open(os.path.join(ROOT, "include", "dm_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return set(re.findall(r"\b(dm_[a-z0-9_]+)\s*\(", text))


def test_header_symbols_exported():
    import __graft_entry__ as entry
    entry.build()                                   # no-op when the in-tree library is current
    from delta_matching_b200 import _lib
    names = _declared()
    assert {"dm_fwd", "dm_delta", "dm_bwd", "dm_quant_qkv", "dm_quant_do", "dm_version"} <= names
    L = _lib.lib()
    for n in names:
        assert hasattr(L, n), n
    assert set(_lib.SIGNATURES) == names
    assert L.dm_version() >= 100
    assert L.dm_numerics() == b"sm100-mx"
    assert os.path.basename(_lib.loaded_library()).startswith("libdm_b200")


def test_argument_checks_without_gpu():
    """Shape validation happens before any CUDA call, so it can be exercised on a machine without a GPU."""
    from delta_matching_b200 import _lib
    L = _lib.lib()
    assert L.dm_quant_qkv_workspace_bytes(4, 4096, 8, 128) == 4 * 8 * 64 * 128 * 4
    assert L.dm_quant_qkv_workspace_bytes(0, 4096, 8, 128) == 0
    rc = L.dm_fwd(None, None, None, None, None, None, 1, 256, 2, 2, 96, 1, None, 0, 0, 0, None, None, None)
    assert rc == -1 and "head_dim" in _lib.last_error()
    rc = L.dm_delta(None, None, None, None, None, None, None, None, None, 1, 256, 3, 2, 128, 1, None, None, None)
    assert rc == -1 and "nheads" in _lib.last_error()
    rc = L.dm_fwd(None, None, None, None, None, None, 70000, 256, 1, 1, 128, 1, None, 0, 0, 0, None, None, None)
    assert rc == -1 and "65535" in _lib.last_error()


@pytest.mark.parametrize("bad", [None, 0x1008], ids=["null", "misaligned"])
def test_whole_pass_entry_points_refuse_bad_pointers(bad):
    """Every buffer of dm_attn_fwd / dm_attn_bwd in turn NULL or 8 bytes off, before any CUDA call; the fine ones are made-up
    addresses that a machine without a GPU never gets to use."""
    from delta_matching_b200 import _lib
    L = _lib.lib()
    fine = 0x10000
    st, shape = (256 * 256, 128, 256), (1, 256, 2, 2, 128, 1)
    names = ("q", "k", "v", "q8", "k8", "v8", "q scales", "k scales", "v scales", "kmean", "workspace", "o", "lse")
    for i, name in enumerate(names):
        p = [bad if j == i else fine for j in range(13)]
        assert L.dm_attn_fwd(p[0], *st, p[1], *st, p[2], *st, *shape, *p[3:], None, None) == -1
        assert f" {name} " in _lib.last_error()
    names = ("d_o", "q8", "k8", "v8", "q scales", "k scales", "v scales", "lse", "do8", "dO scales", "delta", "dq", "dk", "dv", "workspace", "o")
    ws = L.dm_attn_bwd_workspace_bytes(*shape)
    for i, name in enumerate(names):
        if name == "o" and bad is None:                 # no O: the matched delta
            continue
        p = [bad if j == i else fine for j in range(16)]
        assert L.dm_attn_bwd(p[0], *st, p[15], *p[1:11], *shape, *p[11:15], ws, 0, None, None) == -1
        assert f" {name} " in _lib.last_error()


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from delta_matching_b200 import _lib
    monkeypatch.setenv("DM_SO", str(tmp_path / "nope.so"))
    with pytest.raises(RuntimeError, match="does not exist"):
        _lib.library_path()
