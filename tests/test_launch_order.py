"""Launches of several host threads, on the CPU: the native calls, streams and events are fakes that write a log.

What has to hold: the context that a native call reads is its own, and a launch on another stream comes entirely after
the launch before it, so that it can wait for that launch's end (two single-pass grids that overlap on a device can wait
for one another)."""
import threading
import weakref
from types import SimpleNamespace

import pytest
import torch

from fast_sequential_scan_b200 import _lib, sequential_scan_cuda as native, workspace

LIMIT = 5.0      # seconds any wait of a test may take


@pytest.fixture
def fake(monkeypatch):
    """One fake device.  ``stream`` is the calling thread's stream; ``log`` what the host asked of the device, in order;
    ``on_launch(context)`` runs inside a native call."""
    state = SimpleNamespace(log=[], on_launch=lambda ctx: None, thread=threading.local())

    class Event:
        def record(self, stream):
            self.stream = stream.handle
            state.log.append(("record", stream.handle))

    class Stream:
        def __init__(self, handle):
            self.handle = handle

        def wait_event(self, event):
            state.log.append(("wait", self.handle, event.stream))

    class Workspace(workspace.Workspace):
        def __init__(self, device, handle):
            self.device, self.stream_handle, self.buf, self.contexts, self._event = device, handle, None, {}, None
            self.status, self._flag = torch.zeros(1, dtype=torch.int32), [0]
            self.order = workspace._devices.setdefault(device.index, workspace._DeviceOrder())

        def stream(self):
            return Stream(self.stream_handle)

        def ensure(self, nbytes):
            self.buf, self.contexts = torch.zeros(nbytes, dtype=torch.uint8), {}

    def scan(ctx, *args):
        ctx = ctx._obj
        state.on_launch(ctx)
        state.log.append(("launch", ctx.stream, ctx.flags))
        return 0

    monkeypatch.setattr(workspace, "_cache", {})
    monkeypatch.setattr(workspace, "_devices", {})
    monkeypatch.setattr(workspace, "Workspace", Workspace)
    monkeypatch.setattr(workspace, "current_stream_handle", lambda device: state.thread.stream)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(_lib, "lib", lambda: SimpleNamespace(fss_scan_forward_ex=scan, fss_workspace_bytes=lambda *a: 4096))
    monkeypatch.setattr(native, "_view", lambda t: _lib.View(0, 0, 0))
    return state


def _scan(fake, stream, flags=0):
    fake.thread.stream = stream
    t = SimpleNamespace(shape=(1, 4, 8), device=torch.device("cuda", 0))
    native._launch_forward(t, t, t, _lib.DTYPE_F32, _lib.ALGO_AUTO, flags, None)


def _second_thread(target):
    """Starts ``target`` in a thread and gives it time to run as far as it can."""
    thread = threading.Thread(target=target)
    thread.start()
    thread.join(0.2)
    return thread


def test_a_launch_reads_a_context_of_its_own(fake):
    other = []

    def on_launch(ctx):
        before = bytes(ctx)
        if not other:
            other.append(_second_thread(lambda: _scan(fake, 1, _lib.FLAG_REVERSE)))
        assert bytes(ctx) == before
    fake.on_launch = on_launch
    _scan(fake, 1, _lib.FLAG_CONTINUATION)
    other[0].join(LIMIT)
    assert fake.log == [("launch", 1, _lib.FLAG_CONTINUATION), ("launch", 1, _lib.FLAG_REVERSE)]


def test_another_threads_stream_waits_for_the_launch_that_is_under_way(fake):
    other = []

    def on_launch(ctx):
        if not other:
            other.append(_second_thread(lambda: _scan(fake, 2)))
    fake.on_launch = on_launch
    _scan(fake, 1)
    other[0].join(LIMIT)
    _scan(fake, 1)
    assert fake.log == [("launch", 1, 0), ("record", 1), ("wait", 2, 1), ("launch", 2, 0), ("record", 2),
                        ("wait", 1, 2), ("launch", 1, 0), ("record", 1)]


def test_what_the_cpp_functions_hold_is_theirs_until_they_have_launched(fake):
    fake.thread.stream = 1
    ctx, address, release, ws = native._acquire(0, 1, 4, 8, _lib.DTYPE_F32, 0)
    other = _second_thread(lambda: _scan(fake, 2, _lib.FLAG_REVERSE))
    assert fake.log == []
    assert (ctx.stream, ctx.algo, ctx.flags, ws) == (1, _lib.ALGO_AUTO, 0, None)
    assert bytes(_lib.ScanCtx.from_address(address)) == bytes(ctx)
    fake.log.append(("launch", 1, 0))
    release()
    other.join(LIMIT)
    assert fake.log == [("launch", 1, 0), ("record", 1), ("wait", 2, 1), ("launch", 2, _lib.FLAG_REVERSE), ("record", 2)]
    # from the second stream on, every launch is recorded before the lock is given back
    *_, release, ws = native._acquire(0, 1, 4, 8, _lib.DTYPE_F32, 0)
    assert ws is not None
    workspace.launched(ws)
    release()
    assert fake.log[-2:] == [("wait", 1, 2), ("record", 1)]


def test_a_call_that_fails_gives_the_device_back(fake, monkeypatch):
    def broken(ctx):
        raise KeyboardInterrupt
    fake.on_launch = broken
    with pytest.raises(KeyboardInterrupt):
        _scan(fake, 1)
    monkeypatch.setattr(native, "default_algo", lambda: 1 // 0)
    with pytest.raises(ZeroDivisionError):
        native._acquire(0, 1, 4, 8, _lib.DTYPE_F32, 0)
    fake.on_launch = lambda ctx: None
    thread = _second_thread(lambda: _scan(fake, 1))
    thread.join(LIMIT)
    assert not thread.is_alive() and fake.log[-1] == ("launch", 1, 0)


def test_a_replaced_buffer_outlives_the_graphs_that_may_write_to_it(monkeypatch):
    """A captured launch keeps the address of its workspace.  Growing replaces the buffer, and must not free the old one."""
    cleared = []

    def init(address, nbytes, stream):
        cleared.append((address, nbytes))
        return 0
    monkeypatch.setattr(_lib, "lib", lambda: SimpleNamespace(fss_workspace_init=init))
    monkeypatch.setattr(torch.Tensor, "pin_memory", lambda self: self)
    monkeypatch.setattr(workspace, "_devices", {})
    ws = workspace.Workspace(SimpleNamespace(type="cpu", index=0), 1)
    monkeypatch.setattr(ws, "device", torch.device("cpu"))
    made = []
    for nbytes in (1000, 1 << 16, (1 << 16) + 1, 1 << 20, 5000, 1 << 21):
        if ws.buf is None or ws.buf.numel() < nbytes:
            ws.ensure(nbytes)
            made.append(weakref.ref(ws.buf))
    buffers = [ref() for ref in made]
    assert len(buffers) == 4 and all(t is not None for t in buffers)
    assert sum(t.numel() for t in buffers[:-1]) < buffers[-1].numel()
    assert cleared == [(t.data_ptr(), t.numel()) for t in buffers]
    # a launch that reported a failure may have been any of theirs: all are cleared
    cleared.clear()
    ws._flag[0] = 1
    with pytest.raises(RuntimeError):
        ws.raise_if_flagged()
    assert sorted(cleared) == sorted((t.data_ptr(), t.numel()) for t in buffers)
