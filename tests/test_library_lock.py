"""The lock around the library handle and the default contexts may be met again by
the thread that holds it: the garbage collector can run there and close a Context
that was kept in a reference cycle (an exception's traceback, for one)."""
import gc
import threading

from naivedynamics import _lib


class _Cycle:
    """Garbage in a cycle whose finaliser uses the library, as Context's does."""

    def __init__(self):
        self.me = self

    def __del__(self):
        _lib.lib()


def _held():
    with _lib._lock:
        _Cycle()
        gc.collect()


def test_collector_may_close_contexts_under_the_lock(nd):
    t = threading.Thread(target=_held, daemon=True)
    t.start()
    t.join(20.0)
    assert not t.is_alive()


def test_default_context_is_one_per_device(nd, monkeypatch):
    made = []

    class Fake:
        def __init__(self, device=0):
            made.append(device)

    monkeypatch.setattr(_lib, "Context", Fake)
    monkeypatch.setattr(_lib, "_default", {})
    got = []
    ts = [threading.Thread(target=lambda: got.append(_lib.default_context(0))) for _ in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(20.0)
    assert len(got) == 8 and all(c is got[0] for c in got)
