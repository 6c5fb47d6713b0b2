"""Sums whose passes would hold few terms, on registers on both sides of the size from which
those go one Pauli at a time (128 MiB: 23 qubits of complex128, 24 of complex64), and that
such a sum costs no more there than its Paulis one by one."""
from __future__ import annotations

import random
import time

import pytest

pytestmark = pytest.mark.gpu


def _register(nb, n, precision):
    torch = pytest.importorskip("torch")
    s = nb.GpuStateVector(n, precision)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    v = torch.randn(1 << n, 2, generator=g, device="cuda", dtype=torch.float32)
    s.torch_view().copy_(torch.view_as_complex(v / v.norm()))
    torch.cuda.synchronize()
    return s


def _pauli(nb, r, n, letters):
    x = z = 0
    for q in r.sample(range(n), letters):
        x |= 1 << q
        z |= r.randrange(2) << q
    return nb.Pauli(n, x, z, bin(x & z).count("1") & 3)


@pytest.mark.parametrize("n,precision", [(22, 0), (23, 0), (23, 1), (24, 1)])
@pytest.mark.parametrize("count", [2, 3, 9])
def test_scattered_terms_equal_single_paulis(n, precision, count):
    import ncsim_b200 as nb

    s, r = _register(nb, n, precision), random.Random(count)
    terms = [(r.uniform(-1, 1), _pauli(nb, r, n, 9)) for _ in range(count)]
    terms += [(1.0, nb.Pauli(n, terms[0][1].x, 0, 0)), (0.5, nb.Pauli(n, 0, 1 << (n - 1), 0))]
    want = sum(c * s.expectation(p) for c, p in terms)
    # float32 amplitudes are exact in either; every expectation is rounded at 1e-16 of the norm
    assert abs(s.expectation_sum(terms) - want) < 1e-13 * len(terms)


def test_scattered_terms_cost_no_more_than_single_paulis():
    import ncsim_b200 as nb

    n = 27
    s, r = _register(nb, n, 0), random.Random(1)
    terms = [(1.0, _pauli(nb, r, n, 9)) for _ in range(8)]

    def best(f):
        times = []
        for _ in range(7):
            t = time.perf_counter()
            f()
            times.append(time.perf_counter() - t)
        return min(times[2:])

    # in passes of their own they took 1.6 times as long; 1.25 leaves room for the host's noise
    assert best(lambda: s.expectation_sum(terms)) < 1.25 * best(lambda: [s.expectation(p) for _, p in terms])
