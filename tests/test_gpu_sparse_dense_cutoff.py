"""Dense 1-qubit gates of the sparse form whose outputs all stand at the cutoff, so that
rounding decides which of them stay: the step that counts the outputs and the step that
places them have to agree on each one.  On both sides of the one-block form's limit
(4096 entries), one and several key words."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 200])
@pytest.mark.parametrize("m", [300, 4096, 4097, 30000])
def test_outputs_at_the_cutoff_are_counted_and_placed_alike(n, m):
    import ncsim_b200 as nb

    r = np.random.default_rng(m + n)
    q, theta = 20, 1.1
    keys = sorted(set(int(k) for k in r.integers(0, 1 << 39, 2 * m) & ~(1 << q)))[:m]  # no partners
    phase = np.exp(2j * np.pi * r.random(len(keys)))
    s = nb.GpuSparseVector.from_entries(n, keys, phase)
    c, t = math.cos(theta / 2), math.sin(theta / 2)  # the outputs' magnitudes with bit q = 0 and 1
    cutoff = c
    s.with_cutoff(cutoff)
    s.run(nb.Circuit.parse(f"QUBITS {n}\nRY({theta!r}) {q}\n"), nb.StdRng(1))
    got_keys, got = s.entries()
    got_keys = [int(k) for k in got_keys]
    assert all(a < b for a, b in zip(got_keys, got_keys[1:]))
    want = dict(zip(keys, phase))
    assert t < cutoff * (1 - 1e-9)  # those are dropped
    assert set(got_keys) <= set(want)
    # rounding keeps some and drops some: a rounded |a|^2 is on either side about as often
    assert 0.1 * len(keys) < len(got_keys) < 0.98 * len(keys)
    # each part of a product is rounded to 2^-53 of its size
    assert max(abs(v - c * want[k]) for k, v in zip(got_keys, got)) < 4 * 2.0**-53
