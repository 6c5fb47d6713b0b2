"""The stream and buffers that released sparse states leave for the next ones: results
do not depend on reuse, several threads make and release states at once, trimming gives
everything back while states are alive, and a fresh state's timer is not a used one."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circuit(nb, n, k):
    return nb.Circuit.parse(f"QUBITS {n}\n" + "".join(f"H {q}\n" for q in range(k)) + f"CX 0 {n - 1}\nT {n - 1}\nM 1\n")


def test_states_reuse_sets():
    import ncsim_b200 as nb

    errors = []

    def work(t):
        try:
            for i in range(30):
                n, k = (20, 3 + (t + i) % 5) if i % 2 else (300, 2 + (t + i) % 4)
                s = nb.GpuSparseVector(n)
                s.run(_circuit(nb, n, k), nb.StdRng(i))
                assert s.num_entries() == 1 << (k - 1)
                del s
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors
    keep = nb.GpuSparseVector(20)
    many = [nb.GpuSparseVector(20) for _ in range(20)]
    del many  # more than are kept
    nb.trim_memory()
    keep.run(_circuit(nb, 20, 4), nb.StdRng(1))
    assert keep.num_entries() == 8
    a = keep.clone()
    assert np.array_equal(a.entries()[1], keep.entries()[1])


def test_a_reused_set_has_no_started_timer():
    import ncsim_b200 as nb

    a = nb.GpuSparseVector(8)
    a.timer_start()
    assert a.timer_stop() >= 0.0
    del a
    b = nb.GpuSparseVector(8)
    with pytest.raises(nb.SimError):
        b.timer_stop()
