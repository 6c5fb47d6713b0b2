"""Tiled passes at the edges of their tiles and windows: registers below, at and
above one tile (2^11 amplitudes), above the size from which a window keeps the two
lowest qubits, gates whose fixed bits lie in the cube, in the tile and outside the
window, exchanges across one, two and three tile bits, every class of 1-qubit
matrix.  A run gives the gate-by-gate kernels' amplitudes bit for bit."""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ONE = ["H", "RY(1.3)", "RX(0.37)", "SQRT_Y", "SQRT_Y_DAG", "SQRT_X", "SQRT_X_DAG", "S", "S_DAG", "T", "Z", "X", "Y",
       "RZ(2.1)", "PHASE(3,4)"]
TWO = ["CX", "CY", "CZ", "SWAP", "CS", "CS_DAG", "CPHASE(1,3)"]


def _text(n, gates, seed):
    r = random.Random(seed)
    lines = [f"QUBITS {n}"]
    for q in range(n):
        lines.append(f"{ONE[q % 5]} {q}")
    for _ in range(gates):
        u = r.random()
        if u < 0.5:
            lines.append(f"{r.choice(ONE)} {r.randrange(n)}")
        elif u < 0.8:
            lines.append(f"{r.choice(TWO)} {' '.join(map(str, r.sample(range(n), 2)))}")
        elif u < 0.9:
            lines.append(f"{r.choice(['CCX', 'CCZ'])} {' '.join(map(str, r.sample(range(n), 3)))}")
        elif u < 0.94:  # x -> x ^ 7 with phases: an exchange across three bits
            lines.append(f"MONOMIAL(1,2,4;7;3;0;{r.choice(['', '1:1;3:2,4;'])}0,0,0) {' '.join(map(str, r.sample(range(n), 3)))}")
        elif u < 0.97:
            lines.append(f"DIAG(3;1;1:1;3:2,4;5:1,2,4) {' '.join(map(str, r.sample(range(n), 3)))}")
        else:  # on more than ten qubits: a phase polynomial of the index
            qs = r.sample(range(n), n) if n < 12 else r.sample(range(n), 11)
            lines.append(f"DIAG(4;3;5:1;3:6,{1 << (len(qs) - 1)}) {' '.join(map(str, qs))}")
    return "\n".join(lines) + "\n"


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [8, 9, 11, 12, 13, 18, 19, 22])
def test_runs_equal_gate_by_gate(n, precision):
    import ncsim_b200 as nb

    c = nb.Circuit.parse(_text(n, 240, 7 * n + precision))
    got = []
    for passes in (False, True):
        s = nb.GpuStateVector.basis_state(n, 5, precision)
        s.set_tile_passes(passes)
        s.run(c, nb.StdRng(0))
        got.append(s.to_vector())
    assert np.array_equal(got[0], got[1])
