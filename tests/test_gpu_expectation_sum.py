"""Sums of Pauli expectations in shared passes: X parts inside one window, in
several windows and wider than a window, registers below, at and above a tile (2^11
amplitudes), more terms than a pass holds, every phase (Hermitian or not), repeated
terms, both precisions.  Every term and the sum against the single-Pauli kernels."""
from __future__ import annotations

import random

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(nb, n, precision, seed):
    r = np.random.default_rng(seed)
    v = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    return nb.GpuStateVector.from_amplitudes(v / np.linalg.norm(v), precision)


def _terms(nb, n, seed):
    r = random.Random(seed)
    out = []
    for q in range(n - 1):
        out += [(1.0, nb.Pauli(n, 3 << q, 0, 0)), (0.5, nb.Pauli(n, 3 << q, 3 << q, 2)), (0.3, nb.Pauli(n, 0, 3 << q, 0))]
    for _ in range(70):
        out.append((complex(r.uniform(-1, 1), r.uniform(-1, 1)),
                    nb.Pauli(n, r.randrange(1 << n) & r.randrange(1 << n), r.randrange(1 << n), r.randrange(4))))
    full = (1 << n) - 1
    out += [(1.0, nb.Pauli(n, 0, 0, k)) for k in range(4)] + [(1j, nb.Pauli(n, full, full, 1)), (1.0, nb.Pauli(n, full, 0, 0))]
    out += [(0.2, nb.Pauli(n, 0, r.randrange(1 << n), 0)) for _ in range(60)] + out[:3]
    return out


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [3, 7, 8, 9, 10, 11, 12, 13, 17, 20])
def test_sum_equals_single_paulis(n, precision):
    import ncsim_b200 as nb

    s = _state(nb, n, precision, n)
    terms = _terms(nb, n, n)
    single = [s.expectation(p) for _, p in terms]
    for k, (c, p) in enumerate(terms):
        if k % 7 == 0:  # one term through the shared pass, beside a known one
            got = s.expectation_sum([(1.0, p), (2.0, nb.Pauli(n, 0, 0, 0))]) - 2.0 * s.norm_sq().real
            assert abs(got - single[k]) < 1e-13
    want = sum(c * e for (c, _), e in zip(terms, single))
    # every expectation is rounded at 1e-16 of the norm, in another order
    assert abs(s.expectation_sum(terms) - want) < 1e-13 * len(terms)


def test_out_of_register_term_is_refused():
    import ncsim_b200 as nb

    s = nb.GpuStateVector.plus_state(9)
    with pytest.raises(nb.SimError):
        s.expectation_sum([(1.0, nb.Pauli(9, 1, 0, 0)), (1.0, nb.Pauli(9, 1 << 9, 0, 0))])
    assert s.expectation_sum([]) == 0
