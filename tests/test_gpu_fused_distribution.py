"""The fused form gives a tile the same bits however many tiles a register has: one per SM with SMs
to spare, two or four per CTA, sets with a short or absent last share.  A circuit on the 13 lowest
qubits acts on a block of a larger register, picked by its upper index bits, as on a register of 13
qubits; every other amplitude stays zero.
"""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LOW = 13


def _lines(depth, seed):
    r = random.Random(seed)
    out = []
    for _ in range(depth):
        for q in range(LOW):
            out.append("%s %d" % (r.choice(["H", "T", "S", "SQRT_X", "RZ(%r)" % r.uniform(0, 6), "RX(0.4)"]), q))
        for _ in range(LOW // 2):
            out.append("%s %d %d" % (r.choice(["CZ", "CZ", "CX", "CPHASE(1,4)"]), *r.sample(range(LOW), 2)))
    return "\n".join(out) + "\n"


@pytest.mark.parametrize("n", [14, 19, 20, 21, 22])
def test_fused_bits_do_not_depend_on_the_distribution(nb, n):
    r = np.random.default_rng(n)
    v = r.normal(size=1 << LOW) + 1j * r.normal(size=1 << LOW)
    v = (v / np.linalg.norm(v)).astype(np.complex64).astype(np.complex128)
    text = _lines(8, n)
    small = nb.GpuStateVector.from_amplitudes(v, nb.C64)
    _, plan = small.run_fused(nb.Circuit.parse("QUBITS %d\n" % LOW + text), nb.StdRng(0))
    assert plan.passes >= 2 and plan.diagonal_terms > 0
    first = int(r.integers(1 << (n - LOW))) << LOW
    amps = np.zeros(1 << n, dtype=np.complex128)
    amps[first : first + (1 << LOW)] = v
    large = nb.GpuStateVector.from_amplitudes(amps, nb.C64)
    large.run_fused(nb.Circuit.parse("QUBITS %d\n" % n + text), nb.StdRng(0))
    got = large.to_vector()
    assert np.array_equal(got[first : first + (1 << LOW)], small.to_vector())
    got[first : first + (1 << LOW)] = 0
    assert not np.any(got)
