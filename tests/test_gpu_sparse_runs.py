"""Runs of one-to-one ops of the sparse form on 32-entry groups: entry counts
around a warp's 32 entries and a block's, registers around the 32- and 64-qubit
words of a key, every op a run can hold (controlled NOTs, exchanges, affine maps,
phase terms of one to many factors, multi-bit parities, phases of up to 8 and of
more bits, arbitrary phases, Paulis of noise), runs longer than one staged chunk,
and lists of NOTs that end on every place of their four-op groups.  The entries
(keys bit for bit and in order, amplitudes within 1e-12) are those of the same
gates applied one by one, which keep their own kernels."""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gates(n, count, seed):
    r = random.Random(seed)
    out = []
    for i in range(count):
        u = r.random()
        q = lambda k: r.sample(range(n), k)  # noqa: E731
        if u < 0.3:
            for _ in range(r.randrange(1, 10)):
                name, k = r.choice([("X", 1), ("CX", 2), ("CCX", 3), ("SWAP", 2)])
                out.append((name, q(k)))
        elif u < 0.5:
            name, k = r.choice([("Z", 1), ("S", 1), ("T_DAG", 1), ("Y", 1), ("CZ", 2), ("CY", 2), ("CS", 2), ("CCZ", 3),
                                ("PHASE(5,4)", 1), ("CPHASE(3,7)", 2), ("PHASE(77,12)", 1), ("RZ(0.7)", 1)])
            out.append((name, q(k)))
        elif u < 0.6:
            out.append(("MONOMIAL(1,3,4;2;2;0;1:1;3:2,4;0,0,0)", q(3)))
        elif u < 0.7:
            out.append(("MONOMIAL(2,1,4,12,16;9;3;1;5:3;2:1,2,4,8;7:24,3;0,1,3)", q(5)))
        elif u < 0.8:
            out.append(("DIAG(3;1;1:1;3:2,4;5:1,2,8;7:7;2:3,12)", q(4)))
        elif u < 0.9:
            k = min(n, r.choice([11, 40]))
            terms = "".join(f";{r.randrange(1, 8)}:{','.join(str(1 << v) for v in r.sample(range(k), r.randrange(1, 4)))}"
                            for _ in range(r.choice([3, 40, 70])))
            out.append((f"DIAG(3;0{terms})", q(k)))
        else:
            k = min(n, 12)
            out.append((f"DIAG(11;3;5:1;1030:6,{1 << (k - 1)};9:513,12,2)", q(k)))
    return out


@pytest.mark.parametrize("n,inputs", [(17, 0), (17, 3), (31, 5), (32, 6), (33, 5), (63, 7), (64, 9), (65, 5), (128, 4),
                                      (257, 6), (1000, 5), (40, 14)])
def test_run_equals_gate_by_gate(n, inputs):
    import ncsim_b200 as nb

    gates = _gates(n, 160 if inputs < 14 else 40, 31 * n + inputs)
    head = [("H", [q]) for q in range(inputs)]
    lines = [f"{g} {' '.join(map(str, qs))}" for g, qs in head + gates]
    a = nb.GpuSparseVector(n)
    a.run(nb.Circuit.parse(f"QUBITS {n}\n" + "\n".join(lines) + "\n"), nb.StdRng(1))
    b = nb.GpuSparseVector(n)
    for g, qs in head + gates:
        b.apply_gate(nb.Gate.parse(g, len(qs)), qs)
    ka, va = a.entries()
    kb, vb = b.entries()
    assert len(ka) == 1 << inputs
    assert list(ka) == list(kb)
    assert np.abs(va - vb).max() < 1e-12
