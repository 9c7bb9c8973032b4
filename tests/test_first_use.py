"""The library on first use: published when it is ready, whoever asks for it."""
import ctypes
import importlib.util
import os
import shutil
import subprocess
import sys
import sysconfig
import threading
import time

import pytest
import torch


class Calls:
    """Stands in for the native module."""

    def __init__(self, on_bind):
        self.on_bind = on_bind

    def bind(self, *addresses):
        self.on_bind()


@pytest.fixture
def unloaded(dtattn, monkeypatch):
    """As before the first use, with a native module whose bind does what the test says."""
    def prepare(on_bind):
        monkeypatch.setattr(dtattn, "_lib", None)
        monkeypatch.setattr(dtattn, "_calls", Calls(on_bind))
        monkeypatch.setattr(dtattn, "_load_calls", lambda: Calls(on_bind), raising=False)
    return prepare


def test_a_second_thread_waits_for_the_first(dtattn, unloaded):
    bound, early = [], []

    def slowly():
        time.sleep(0.3)
        bound.append(True)

    def use():
        dtattn.lib().dt_abi_version()
        early.append(not bound)

    unloaded(slowly)
    threads = [threading.Thread(target=use) for _ in range(4)]
    for t in threads:
        t.start()
        time.sleep(0.03)
    for t in threads:
        t.join()
    assert early == [False] * 4 and bound == [True]


def test_a_failure_is_not_taken_for_a_library(dtattn, unloaded):
    def fails():
        raise OSError("no such symbol")

    unloaded(fails)
    for _ in range(2):
        with pytest.raises(OSError):
            dtattn.lib()
    assert dtattn._lib is None


def test_the_native_module_calls_nothing_before_it_is_bound(dtattn):
    child = """
import importlib.util, sys, torch
spec = importlib.util.spec_from_file_location("dtattn_calls", sys.argv[1])
module = importlib.util.module_from_spec(spec)
spec.loader.exec_module(module)
print("RESULT", module.run(bytes(int(sys.argv[2])), None, 0, 0, 0))
"""
    r = subprocess.run([sys.executable, "-c", child, dtattn._calls.__file__, str(ctypes.sizeof(dtattn.SdpaParams))],
                       capture_output=True, text=True, cwd=os.path.dirname(os.path.abspath(__file__)))
    assert r.returncode == 0 and "RESULT None" in r.stdout, r.stderr


def test_importing_needs_no_build(dtattn, tmp_path):
    """What calls no kernel works from the sources alone; the first use of the library says what is missing."""
    shutil.copytree(os.path.dirname(dtattn.__file__), tmp_path / "pkg" / "dtattn", ignore=shutil.ignore_patterns("__pycache__"))
    child = """
import os, sys
sys.path.insert(0, sys.argv[1])
import dtattn
from dtattn import selection, sharding
assert os.path.dirname(dtattn.__file__).startswith(sys.argv[1])
dtattn.SdpaParams()
for library in (dtattn.LIB_PATH, sys.argv[2]):  # neither is there; only the native module is missing
    dtattn.LIB_PATH = library
    for _ in range(2):
        try:
            dtattn.lib()
        except ImportError as e:
            print("RESULT", str(e).split()[0])
"""
    r = subprocess.run([sys.executable, "-c", child, str(tmp_path / "pkg"), dtattn.LIB_PATH], capture_output=True, text=True)
    said = [os.path.basename(line.split()[1]) for line in r.stdout.splitlines() if line.startswith("RESULT")]
    assert r.returncode == 0 and [x.startswith("libdtattn") for x in said] == [True, True, False, False], (said, r.stderr)
    assert all("dtattn_calls" in x for x in said[2:])


def test_a_module_built_for_another_torch_is_not_loaded(dtattn, monkeypatch):
    """Neither loaded nor taken for up to date: the torch and the Python that it is compiled against are in its name."""
    spec = importlib.util.spec_from_file_location("dt_build", os.path.join(os.path.dirname(dtattn.__file__), "..", "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    here = build.build_calls()
    assert os.path.samefile(here, dtattn._calls.__file__)
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert not os.path.exists(build.calls_path())
    with pytest.raises(ImportError, match="torch0.0.1"):
        dtattn._load_calls()
    monkeypatch.undo()
    monkeypatch.setattr(sysconfig, "get_config_var", lambda name: "cpython-000")
    with pytest.raises(ImportError, match="cpython-000"):
        dtattn._load_calls()
