"""A host thread keeps the buffers that sparse runs are built in from one circuit to the next,
small ones only: what a long circuit's runs took is given back with the call."""
from __future__ import annotations

import ctypes
import gc

import pytest

pytestmark = pytest.mark.gpu


def _resident():
    gc.collect()
    ctypes.CDLL(None).malloc_trim(0)  # what is free, as the parser's text, does not count
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * 4096


@pytest.mark.parametrize("n", [40, 100])
def test_long_runs_leave_no_large_buffers(n):
    import ncsim_b200 as nb

    k = 40
    terms = "".join(f";{1 + j % 7}:{1 << (j % k)},{1 << (j * 7 % k)}" for j in range(400))
    long = nb.Circuit.parse(f"QUBITS {n}\nX 0\n" + f"DIAG(3;0{terms}) {' '.join(map(str, range(k)))}\nCX 0 1\n" * 4000)
    short = nb.Circuit.parse(f"QUBITS {n}\nX 0\nCX 0 1\nT 0\n")
    rng = nb.StdRng(1)
    nb.GpuSparseVector.zero_state(n).run(short, rng)
    before = _resident()
    nb.GpuSparseVector.zero_state(n).run(long, rng)  # a stream of 13 MB, and its copy for the upload
    assert _resident() - before < 10 << 20
