"""scene.recording without a GPU: what it calls, in what order, from two threads."""
import contextlib
import gc
import threading
from types import SimpleNamespace


def test_no_thread_synchronises_the_device_while_another_records(monkeypatch):
    """A device synchronisation ends a recording that is under way.  Two threads record at the same time: the second one's
    synchronisation waits for the first one's recording to end, and the collector is as it was afterwards."""
    import torch
    from heatflow_mpm import scene
    events, inside, second = [], threading.Event(), threading.Event()

    def synchronize(device):
        events.append(("sync", threading.current_thread().name))
        if threading.current_thread().name == "b":
            second.set()

    monkeypatch.setattr(torch.cuda, "synchronize", synchronize)
    monkeypatch.setattr(torch.cuda, "stream", lambda s: contextlib.nullcontext())

    def record():
        name = threading.current_thread().name
        graph = SimpleNamespace(capture_begin=lambda **kw: events.append(("begin", name)),
                                capture_end=lambda: events.append(("end", name)))
        with scene.recording(graph, SimpleNamespace(device="cuda:0")):
            inside.set()
            if name == "a":
                second.wait(0.5)       # the other thread has time to do what it must not

    a, b = (threading.Thread(target=record, name=nm) for nm in "ab")
    collecting = gc.isenabled()
    a.start()
    assert inside.wait(5.0)
    b.start()
    a.join(5.0)
    b.join(5.0)
    assert events == [(what, who) for who in "ab" for what in ("sync", "begin", "end")]
    assert gc.isenabled() == collecting
