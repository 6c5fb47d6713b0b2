"""Calls that had no device memory of their own to ask for still ask for none: they work
on the state's scratch, whatever is left of the device's memory."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


def test_expectation_sum_takes_nothing_from_the_pool():
    import ncsim_b200 as nb

    n = 14
    s = nb.GpuStateVector.plus_state(n)
    # more passes and terms than one fill of the scratch: every X part of weight up to 3 in many windows
    terms = [(1.0, nb.Pauli(n, x, z, 0)) for x in range(1 << 10) for z in (0, 1 << 12, 5 << 10)]
    terms += [(0.5, nb.Pauli(n, x << 4, 0, 0)) for x in range(1 << 10)] * 14  # repeated: 14336 terms more
    s.expectation(terms[0][1])
    nb.trim_memory()
    before = nb.pool_info()
    got = s.expectation_sum(terms)
    assert nb.pool_info() == before
    # <+|P|+> is 1 without Z and 0 with it
    assert abs(got - ((1 << 10) + 0.5 * 14 * (1 << 10))) < 1e-9


@pytest.mark.parametrize("n", [1, 12])
def test_measurements_of_a_run_take_nothing_from_the_pool(n):
    import ncsim_b200 as nb

    c = nb.Circuit.parse(f"QUBITS {n}\nH 0\nM 0\nR 0\nH 0\nMPP X0\n")
    s, rng = nb.GpuStateVector(n), nb.StdRng(1)
    nb.trim_memory()
    before = nb.pool_info()
    assert s.run(c, rng)[1] is False  # |+> measured in X
    assert nb.pool_info() == before
