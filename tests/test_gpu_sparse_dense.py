"""Dense 1-qubit gates of the sparse form: entry counts on both sides of the
one-block form's limit (8192 outputs), gates on the lowest, the highest and middle
qubits (first and last key word), pairs with one and with both partners present,
interference that drops entries, a cutoff, unsorted entries before the gate.
Against the dense oracle's amplitudes (small registers) and the oracle's wide
restatement; entries sorted, no zeros."""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DENSE = ["H", "SQRT_X", "SQRT_Y_DAG", "RX(0.9)", "RY(2.2)"]


@pytest.fixture(scope="module")
def oracle():
    from oracle import oracle as O

    O.build()
    return O


@pytest.mark.parametrize("n,seed", [(1, 1), (2, 2), (5, 3), (12, 4), (13, 5), (14, 6), (15, 7)])
def test_dense_layers_against_the_dense_oracle(oracle, n, seed):
    import ncsim_b200 as nb

    r = random.Random(seed)
    lines = [f"QUBITS {n}"]
    for layer in range(3):
        for q in r.sample(range(n), n):
            lines.append(f"{r.choice(DENSE)} {q}")
        if layer == 0:  # leaves the entries unsorted
            lines += [f"X {r.randrange(n)}", f"RZ(0.3) {r.randrange(n)}"]
            if n > 1:
                lines.append(f"CX {' '.join(map(str, r.sample(range(n), 2)))}")
    text = "\n".join(lines) + "\n"
    g = nb.GpuSparseVector(n)
    g.run(nb.Circuit.parse(text), nb.StdRng(1))
    o = oracle.StateVector(n)
    o.run(oracle.Circuit(text), oracle.StdRng(1))
    assert np.abs(g.to_vector() - o.to_vector()).max() < 1e-12
    k, v = g.entries()
    assert np.all(np.diff(k.astype(np.int64)) > 0) and np.all(v != 0)


def test_interference_drops_exact_zeros():
    import ncsim_b200 as nb

    n = 13
    g = nb.GpuSparseVector(n)
    g.run(nb.Circuit.parse(f"QUBITS {n}\n" + "".join(f"H {q}\n" for q in range(n))), nb.StdRng(1))
    assert g.num_entries() == 1 << n
    g.with_cutoff(1e-10)  # the second Hadamards leave rounding residues where the amplitudes cancel
    g.run(nb.Circuit.parse(f"QUBITS {n}\n" + "".join(f"H {q}\n" for q in reversed(range(n)))), nb.StdRng(1))
    k, v = g.entries()
    assert list(k) == [0] and abs(v[0] - 1) < 1e-12


@pytest.mark.parametrize("n", [64, 65, 256, 257, 1000])
def test_gates_on_every_key_word(oracle, n):
    import ncsim_b200 as nb

    r = random.Random(n)
    qs = [0, n - 1, 63, n // 2, min(64, n - 1)] + r.sample(range(n), 8)
    lines = [f"QUBITS {n}"] + [f"{r.choice(DENSE)} {q}" for q in qs]
    lines += [f"CCX {' '.join(map(str, r.sample(range(n), 3)))}" for _ in range(9)] + [f"H {qs[1]}", f"RY(0.4) {qs[3]}"]
    g = nb.GpuSparseVector(n)
    g.run(nb.Circuit.parse("\n".join(lines) + "\n"), nb.StdRng(1))
    h = nb.GpuSparseVector(n)
    for line in lines[1:]:
        name, *q = line.split()
        h.apply_gate(nb.Gate.parse(name), [int(v) for v in q])
    kg, vg = g.entries()
    kh, vh = h.entries()
    assert list(kg) == list(kh) and np.abs(vg - vh).max() < 1e-12
    if n > 64:
        o = oracle.WideSparse("\n".join(lines) + "\n", 1)
        ok, oa = o.entries()
        assert list(kg) == list(ok) and np.abs(np.asarray(vg) - np.asarray(oa)).max() < 1e-12
