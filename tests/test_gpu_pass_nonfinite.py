"""Tiled passes on registers with infinite and NaN amplitudes, and with amplitudes that
overflow on the way: a run gives what the gates one by one give, part by part (0 * inf is
NaN there, also where a matrix or a phase has zero parts).  Each class of op, registers
below, at and above one tile, exchanges across three bits, both precisions."""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILL = {
    "signs": ["Z {0}", "CZ {0} {1}", "CCZ {0} {1} {2}"],
    "turns": ["S {0}", "S_DAG {0}", "CS {0} {1}", "Z {0}"],
    "phases": ["T {0}", "RZ(0.4) {0}", "CPHASE(1,3) {0} {1}"],
    "moves": ["X {0}", "CX {0} {1}", "SWAP {0} {1}", "CY {0} {1}", "MONOMIAL(1,2,4;7;3;0;0,0,0) {0} {1} {2}"],
    "tables": ["DIAG(3;1;1:1;3:2,4;5:1,2,4) {0} {1} {2}", "Z {0}"],
}
MIX = ["H", "RY(1.3)", "RX(0.37)", "SQRT_Y", "SQRT_X", "SQRT_X_DAG", "SQRT_Y_DAG"]


def _parts(v):
    return np.ascontiguousarray(v).view(np.float64)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [8, 9, 11, 13, 19])
@pytest.mark.parametrize("fill", sorted(FILL))
def test_runs_equal_gate_by_gate(n, precision, fill):
    import ncsim_b200 as nb

    r = random.Random(n)
    odd = [complex(np.inf, 1), complex(-2, np.inf), complex(0, -np.inf), complex(np.nan, 1), complex(3, np.nan), complex(np.inf, 0)]
    huge = 1.5e308 if precision == 0 else 3.3e38  # finite; a sum of two is not
    for mix in MIX + [None]:
        lines = [r.choice(FILL[fill]).format(*r.sample(range(n), 3)) for _ in range(24)]
        if mix:
            lines.insert(12, f"{mix} {r.randrange(n)}")
            lines.insert(20, f"{mix} {r.randrange(n)}")
        c = nb.Circuit.parse(f"QUBITS {n}\n" + "\n".join(lines) + "\n")
        g = np.random.default_rng(n)
        amps = g.normal(size=1 << n) + 1j * g.normal(size=1 << n)
        for v in odd:
            amps[r.randrange(1 << n)] = v
        amps[r.randrange(1 << n)] = 0
        amps[3], amps[3 ^ 1 << (n - 1)] = huge, huge * 1j
        got = []
        for passes in (False, True):
            s = nb.GpuStateVector.from_amplitudes(amps, precision)
            s.set_tile_passes(passes)
            s.run(c, nb.StdRng(0))
            got.append(_parts(s.to_vector()))
        assert not np.isfinite(got[0]).all()
        assert np.array_equal(got[0], got[1], equal_nan=True), (mix, lines)
