"""The native calls and other threads of the interpreter: a call that waits lets them run."""
import ctypes
import os
import subprocess
import threading
import time

import pytest
import torch

FAKE_SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "fake", "slow_calls.c")


@pytest.fixture
def slow_calls(dtattn, tmp_path):
    """The native calls on top of stand-ins that take 0.3 s each."""
    out = tmp_path / "libslow_calls.so"
    subprocess.check_call(["gcc", "-O1", "-shared", "-fPIC", "-o", str(out), FAKE_SRC])
    fake = ctypes.CDLL(str(out))
    address = lambda fn: ctypes.cast(fn, ctypes.c_void_p).value  # noqa: E731
    dtattn._calls.bind(*[address(fake.needs_none if name.endswith("workspace_size") else fake.slow) for name in dtattn._CALLS])
    yield dtattn._calls
    dtattn._calls.bind(*[address(getattr(dtattn.lib(), name)) for name in dtattn._CALLS])


def ticks_during(call):
    """How often another thread comes round (every millisecond at best) while `call` runs."""
    ticks, stop = [], threading.Event()

    def other():
        while not stop.is_set():
            ticks.append(time.monotonic())
            time.sleep(0.001)

    t = threading.Thread(target=other)
    t.start()
    try:
        time.sleep(0.05)
        begin = time.monotonic()
        got = call()
        end = time.monotonic()
    finally:
        stop.set()
        t.join()
    assert end - begin >= 0.3
    return got, sum(begin < x < end for x in ticks)


def test_a_waiting_call_with_scratch(dtattn, slow_calls):
    out = object()
    got, ticks = ticks_during(lambda: slow_calls.run(bytes(ctypes.sizeof(dtattn.SdpaParams)), out, 0, 0, 0))
    assert got is out and ticks > 5


@pytest.mark.gpu
def test_waiting_calls(dtattn, slow_calls):
    x = torch.zeros(1, 4, 2, 64, dtype=torch.float16, device="cuda:0")
    for call in (lambda: dtattn.sdpa_forward(x, x, x, 0.125), lambda: dtattn.qk_prologue(x, x),
                 lambda: dtattn.decode_step(x[:, :1], x, x, x[:, :1], x[:, :1], None, 0.125, 3),
                 lambda: dtattn.sparse_indexed_attention(x, x, x, None, None, None, 0.125)):
        got, ticks = ticks_during(call)
        assert got is not None and ticks > 5
