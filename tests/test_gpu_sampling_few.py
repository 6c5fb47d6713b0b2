"""Few shots: the shots of a call are found by walking their whole blocks or from the parts'
sums, by a rule on their number; either way they are the same indices."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [11, 12, 13, 14])
def test_a_calls_first_shots_are_those_of_a_shorter_call(n, precision):
    import ncsim_b200 as nb

    r = np.random.default_rng(n)
    v = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    v[r.random(1 << n) < 0.3] = 0
    s = nb.GpuStateVector.from_amplitudes(v / np.linalg.norm(v), precision)
    u = np.concatenate([[0.0, 1 - 2.0**-53], r.random(62)])
    r.shuffle(u)
    all_of_them = s.sample_uniforms(u)
    for shots in (1, 2, 3, 4, 5, 8, 9, 16):
        assert np.array_equal(s.sample_uniforms(u[:shots]), all_of_them[:shots])
