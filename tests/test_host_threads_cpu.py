"""State that the op layer keeps per device, first asked for by several host threads at once (no GPU needed: what is asked of
torch is stood in for)."""
import contextlib
import threading
import time

import torch


def test_status_word_is_one_per_device_for_all_threads(monkeypatch):
    """The native route keeps the word's address for good, so a second word for the device must not come to be."""
    from delta_matching_b200 import ops

    class Slow:
        def __init__(self, *a, **kw):
            pass

        def pin_memory(self):
            time.sleep(0.05)                      # a first pinned allocation sets the device up
            return object()

    monkeypatch.setattr(ops, "_STATUS", {})
    monkeypatch.setattr(ops.torch, "zeros", Slow)
    monkeypatch.setattr(ops.torch.cuda, "device", lambda idx: contextlib.nullcontext())
    start, got = threading.Barrier(4), []

    def ask():
        start.wait()
        got.append(ops.status_word(torch.device("cuda", 0)))

    threads = [threading.Thread(target=ask) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 4 and all(w is ops._STATUS[0] for w in got)
