"""The device copy of a fused plan comes from the library's pool and goes back to it with the
circuit: a new circuit's first run maps no memory that an earlier one has left there."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def _text(n, depth):
    lines = [f"QUBITS {n}"]
    for d in range(depth):
        lines += [f"{('H', 'SQRT_X', 'T', 'RZ(0.7)')[(q + d) % 4]} {q}" for q in range(n)]
        lines += [f"CZ {q} {(q + 1 + d) % n}" for q in range(0, n - 1, 2) if (q + 1 + d) % n != q]
    return "\n".join(lines) + "\n"


def test_plans_come_from_the_pool_and_go_back():
    import ncsim_b200 as nb

    n = 16
    s, rng = nb.GpuStateVector(n, nb.C64), nb.StdRng(1)
    nb.trim_memory()
    used = nb.pool_info()["used_bytes"]
    reserved = None
    for depth in (12, 12, 10):
        c = nb.Circuit.parse(_text(n, depth))
        s.run_fused(c, rng)
        assert nb.pool_info()["used_bytes"] > used  # the plan lives with the circuit
        del c
        s.synchronize()
        assert nb.pool_info()["used_bytes"] == used
        if reserved is not None:
            assert nb.pool_info()["reserved_bytes"] == reserved
        reserved = nb.pool_info()["reserved_bytes"]

