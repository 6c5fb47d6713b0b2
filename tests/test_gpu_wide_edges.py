"""Dense gates on 6 to 10 qubits of complex128 registers at the edges of the tensor
kernel's tiles: registers with fewer fibers than a tile is wide, gate qubits at the
bottom (the fibers' amplitudes contiguous), at the top, in the middle and mixed in any
order, every tile shape, against numpy (the sums have 2^k <= 1024 products of unit
vectors' entries, each rounded at 1e-16: 1e-13 covers them)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [6, 7, 8, 9, 10])
@pytest.mark.parametrize("extra", [0, 1, 3, 5, 6, 8])
def test_tiles_and_placements(k, extra):
    import ncsim_b200 as nb

    n = k + extra
    r = np.random.default_rng(100 * k + extra)
    u = np.linalg.qr(r.normal(size=(1 << k, 1 << k)) + 1j * r.normal(size=(1 << k, 1 << k)))[0]
    v = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    v /= np.linalg.norm(v)
    for qs in (list(range(k)), list(range(n - k, n))[::-1], [int(q) for q in r.permutation(n)[:k]]):
        s = nb.GpuStateVector.from_amplitudes(v)
        s.apply_matrix(u, qs)
        t = v.reshape((2,) * n)
        got = np.tensordot(u.reshape((2,) * (2 * k)), t, axes=([2 * k - 1 - j for j in range(k)], [n - 1 - q for q in qs]))
        want = np.moveaxis(got, list(range(k)), [n - 1 - qs[k - 1 - a] for a in range(k)]).reshape(-1)
        assert np.abs(s.to_vector() - want).max() < 1e-13
