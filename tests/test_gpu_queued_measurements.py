"""Runs whose measurements and resets are decided on the device: the record, the
amplitudes and the generator's position afterwards are those of the same ops one
call at a time (`measure`, projections and flips on the host's decisions), on
registers of one block and of many, both precisions, with certain and uncertain
outcomes, Paulis with X and Y parts, more measurements than the queue holds, noise
(which draws) between them, and an op that is refused after a measurement."""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ops(n, count, seed):
    r = random.Random(seed)
    ops = [("gate", "H", [q]) for q in range(n)]
    for _ in range(count):
        u = r.random()
        if u < 0.35:
            ops.append(("gate", r.choice(["H", "T", "SQRT_X", "RY(0.3)", "X"]), [r.randrange(n)]))
        elif u < 0.45 and n > 1:
            ops.append(("gate", "CX", r.sample(range(n), 2)))
        elif u < 0.7:
            ops.append(("M", f"Z{r.randrange(n)}"))
        elif u < 0.8:
            k = r.randrange(1, min(n, 4) + 1)
            ops.append(("MPP", "*".join(f"{r.choice('XYZ')}{q}" for q in r.sample(range(n), k))))
        elif u < 0.92:
            ops.append(("R", r.randrange(n)))
        else:
            ops.append(("noise", r.randrange(n)))
    return ops


@pytest.mark.parametrize("n,count,precision", [(1, 60, 0), (3, 700, 0), (6, 200, 1), (9, 200, 0), (13, 120, 1), (17, 80, 0),
                                               (20, 40, 0)])
def test_run_equals_single_calls(n, count, precision):
    import ncsim_b200 as nb

    ops = [o for o in _ops(n, count, 5 * n + count) if o[0] != "noise"]
    lines = [f"QUBITS {n}"]
    for o in ops:
        if o[0] == "gate":
            lines.append(f"{o[1]} {' '.join(map(str, o[2]))}")
        else:
            lines.append(f"M {o[1][1:]}" if o[0] == "M" else f"{o[0]} {o[1]}")
    a, ra = nb.GpuStateVector(n, precision), nb.StdRng(n)
    rec = a.run(nb.Circuit.parse("\n".join(lines) + "\n"), ra)
    b, rb = nb.GpuStateVector(n, precision), nb.StdRng(n)
    b.set_tile_passes(False)
    want = []
    for o in ops:
        if o[0] == "gate":
            b.apply_gate(nb.Gate.parse(o[1]), o[2])
        elif o[0] == "R":
            if b.measure(nb.Pauli.z_on(n, o[1]), rb):
                b.apply_pauli(nb.Pauli(n, 1 << o[1], 0, 0))
        else:
            want.append(b.measure(nb.Pauli.from_string(n, o[1]), rb))
    assert rec == want
    assert np.array_equal(a.to_vector(), b.to_vector())
    assert ra.next_u64() == rb.next_u64()


@pytest.mark.parametrize("n,seed", [(2, 1), (8, 2), (14, 3)])
def test_noise_between_measurements_matches_the_oracle(n, seed):
    import ncsim_b200 as nb
    from oracle import oracle as O

    O.build()
    lines = [f"QUBITS {n}"]
    for o in _ops(n, 250, seed):
        if o[0] == "gate":
            lines.append(f"{o[1]} {' '.join(map(str, o[2]))}")
        elif o[0] == "noise":
            lines.append(f"DEPOLARIZE1(0.3) {o[1]}")
        else:
            lines.append(f"M {o[1][1:]}" if o[0] == "M" else f"{o[0]} {o[1]}")
    text = "\n".join(lines) + "\n"
    g, r = nb.GpuStateVector(n), nb.StdRng(seed)
    rec = g.run(nb.Circuit.parse(text), r)
    o, ro = O.StateVector(n), O.StdRng(seed)
    assert rec == o.run(O.Circuit(text), ro)
    # 250 ops at 1e-16 each leave the states within 1e-12 of one another after normalising
    va, vo = g.to_vector(), o.to_vector()
    assert np.abs(va / np.linalg.norm(va) - vo / np.linalg.norm(vo)).max() < 1e-12
    assert r.next_u64() == ro.next_u64()


def test_a_refused_op_leaves_the_draws_before_it():
    import ncsim_b200 as nb

    n = 5
    c = nb.Circuit.parse(f"QUBITS {n}\nH 0\nM 0\nH 1\nM 1\n")
    a, ra = nb.GpuStateVector(n), nb.StdRng(3)
    a.run(c, ra)
    rb = nb.StdRng(3)
    rb.gen_f64()
    rb.gen_f64()
    assert ra.next_u64() == rb.next_u64()
