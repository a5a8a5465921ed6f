"""The binding's current-stream handle (gi._stream) from several threads: the first call
sets the fast path up, and a call of another thread at any point of that set-up gets a
handle too.  The other thread is played at every bytecode of the first call."""
import sys
import types

from legitengine_gb300 import gi


def test_a_call_during_the_first_call(monkeypatch):
    stream = types.SimpleNamespace(cuda_stream=77)
    torch = types.SimpleNamespace(
        cuda=types.SimpleNamespace(current_stream=lambda: stream),
        _C=types.SimpleNamespace(_cuda_getCurrentRawStream=lambda device: 70 + device, _cuda_getDevice=lambda: 7))
    monkeypatch.setattr(gi, "_torch", lambda: torch)
    state = [k for k, v in vars(gi).items() if k in ("_raw_stream", "_device", "_current_handle")]
    for k in state:
        monkeypatch.setattr(gi, k, None)
    calls = 0

    def other_thread(frame, event, arg):
        nonlocal calls
        if frame.f_code is not gi._first_stream.__code__:
            return None
        frame.f_trace_opcodes = True
        if event == "opcode":
            saved = {k: getattr(gi, k) for k in state}
            sys.settrace(None)
            try:
                assert gi._stream() == 77
                calls += 1
            finally:
                for k, v in saved.items():
                    setattr(gi, k, v)
                sys.settrace(other_thread)
        return other_thread

    before = sys.gettrace()
    sys._getframe().f_trace_opcodes = True  # Python 3.12 looks for it when tracing starts
    sys.settrace(other_thread)
    try:
        assert gi._stream() == 77
    finally:
        sys.settrace(before)
    assert calls > 5
    assert gi._stream() == 77
