"""An integration's output bytes copied out of the library (correlator._collect):
pieces smaller and larger than a copy thread's share, both result types, and the
copy where no thread can be started any more -- the integration is counted by
then, so its bytes must not be lost."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from sfxc_gpu import correlator

MB = 1 << 20


def pieces(sizes):
    data = [np.random.Generator(np.random.PCG64(n)).integers(0, 256, size=n, dtype=np.uint8) for n in sizes]
    return [(d.ctypes.data if n else 0, n) for d, n in zip(data, sizes)], b"".join(d.tobytes() for d in data), data


@pytest.mark.parametrize("kind", [bytes, bytearray])
@pytest.mark.parametrize("sizes", [[], [0], [1], [0, 7, 5], [8 * MB - 1], [8 * MB], [9 * MB + 3], [3, 41 * MB + 1, 0, 5 * MB]])
def test_pieces_in_order(kind, sizes):
    p, want, keep = pieces(sizes)
    got = correlator._collect(p, kind)
    assert type(got) is kind and got == want


@pytest.mark.parametrize("started", [0, 2])
def test_no_more_threads(monkeypatch, started):
    p, want, keep = pieces([41 * MB + 5])
    start, left = threading.Thread.start, [started]

    def limited(self):
        if not left[0]:
            raise RuntimeError("can't start new thread")
        left[0] -= 1
        start(self)

    monkeypatch.setattr(threading.Thread, "start", limited)
    assert correlator._collect(p, bytes) == want


def test_at_interpreter_exit():
    code = """
import atexit, ctypes as C, sys
from sfxc_gpu import correlator
src = C.create_string_buffer(b"x" * (9 << 20), 9 << 20)
atexit.register(lambda: print(correlator._collect([(C.addressof(src), 9 << 20)], bytes) == src.raw))
"""
    pkg = os.path.dirname(os.path.dirname(correlator.__file__))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                       env=dict(os.environ, PYTHONPATH=pkg))
    assert r.stdout.strip() == "True", r.stderr
