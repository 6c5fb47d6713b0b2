"""The ops of a tiled pass that sweep the tile: phase tables on 1 to 10 qubits, phase
polynomials on more (no term to four, values of 1 to 32 bits, with a scalar), exchanges
across three and more bits (with phases, with several fixed bits), inside and outside the
window, between ops of the chains.  Registers below, at and above one tile.  A run gives
the gate-by-gate kernels' amplitudes bit for bit, and takes about their time at most."""
from __future__ import annotations

import random
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _terms(r, k, bits, count, most=3):
    t = [f"{r.randrange(1, 1 << bits)}:" + ",".join(str(r.randrange(1, 1 << k)) for _ in range(r.randrange(1, most + 1))) for _ in range(count)]
    return "".join(";" + x for x in t)


def _identity(k):
    return ",".join(str(1 << j) for j in range(k))


def _qubits(r, n, k):
    return " ".join(map(str, r.sample(range(n), k)))


def _tables(r, n):
    k = r.randrange(1, min(n, 10) + 1)
    bits = r.choice([1, 2, 3, 6])
    return f"DIAG({bits};{r.randrange(1 << bits)}{_terms(r, k, bits, r.randrange(1, 4))}) {_qubits(r, n, k)}"


def _polynomials(r, n):
    k = r.randrange(11, n + 1)
    bits = r.choice([1, 3, 8, 9, 17, 32])
    terms = _terms(r, k, bits, r.randrange(0, 5), 2)  # at most 8 parities
    if r.random() < 0.4:
        return f"MONOMIAL({_identity(k)};0;{bits};{r.randrange(1 << bits)}{terms};0,{r.randrange(1, 8, 2)},3) {_qubits(r, n, k)}"
    return f"DIAG({bits};{r.randrange(1 << bits)}{terms}) {_qubits(r, n, k)}"


def _exchanges(r, n):
    if r.random() < 0.3:  # two qubits exchanged and a third flipped where they differ: two of three moving bits fixed
        return f"MONOMIAL(2,1,7;0;3;0;0,0,0) {_qubits(r, n, 3)}"
    k = r.randrange(3, min(n, 8) + 1)
    shift = (1 << k) - 1 if r.random() < 0.5 else r.choice([7, (1 << k) - 1 & ~2])
    phase = r.choice(["", ";2:1", ";1:1"])
    return f"MONOMIAL({_identity(k)};{shift};3;{r.choice([0, 0, 3])}{phase};0,0,0) {_qubits(r, n, k)}"


KINDS = {"tables": _tables, "polynomials": _polynomials, "exchanges": _exchanges}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [8, 9, 10, 11, 12, 13, 19])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_runs_equal_gate_by_gate(kind, n, precision):
    import ncsim_b200 as nb

    if kind == "polynomials" and n < 11:
        pytest.skip("polynomials on ten qubits and fewer are tables")
    r = random.Random(100 * n + precision)
    lines = [f"H {q}" for q in range(n)]
    for _ in range(60):
        lines.append(KINDS[kind](r, n) if r.random() < 0.6 else r.choice(["H {0}", "T {0}", "CX {0} {1}", "CZ {0} {1}", "RX(0.3) {1}"])
                     .format(*r.sample(range(n), 2)))
    c = nb.Circuit.parse(f"QUBITS {n}\n" + "\n".join(lines) + "\n")
    got = []
    for passes in (False, True):
        s = nb.GpuStateVector.basis_state(n, 3, precision)
        s.set_tile_passes(passes)
        s.run(c, nb.StdRng(0))
        got.append(s.to_vector())
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("kind", ["tables", "polynomials"])
def test_passes_take_at_most_about_the_time_of_the_gates_one_by_one(kind):
    import ncsim_b200 as nb

    n, r = 20, random.Random(7)
    if kind == "tables":
        lines = [f"DIAG(5;3{_terms(r, 8, 5, 6, 2)}) {_qubits(r, n, 8)}" for _ in range(40)]
    else:
        lines = []
        for _ in range(30):
            lines += [f"DIAG(4;3;5:1;3:6,1024) {_qubits(r, n, 11)}", f"H {r.randrange(n)}"]
    c = nb.Circuit.parse(f"QUBITS {n}\n" + "\n".join(lines) + "\n")
    best = []
    for passes in (False, True):
        s, rng, times = nb.GpuStateVector.plus_state(n), nb.StdRng(0), []
        s.set_tile_passes(passes)
        for _ in range(12):
            t = time.perf_counter()
            s.run(c, rng)
            times.append(time.perf_counter() - t)
        best.append(min(times[3:]))
    assert best[1] < 1.5 * best[0], best  # evaluated in the chains: polynomials 3.6 times
