"""Born sampling with the block search on the device: registers below one block
(4096 amplitudes), of one, a few and many blocks (one, two and three rounds of the
32-way search), both precisions, states with empty blocks and zero amplitudes, draws
of exactly 0 and next to 1.  Every index is that of the rule walked block by block
(block weights, the first running sum above the draw, the walk inside the block)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walked(s, n, u):
    block = min(4096, 1 << n)
    hi = np.array([], dtype=np.float64)
    run = 0.0
    w = s.block_weights(block)
    hi = np.empty_like(w)
    for i, v in enumerate(w):  # the sequential running sum
        run += v
        hi[i] = run
    t = u * run
    b = np.minimum(np.searchsorted(hi, t, side="right"), len(hi) - 1).astype(np.uint64)
    acc = np.where(b > 0, hi[np.maximum(b.astype(np.int64) - 1, 0)], 0.0)
    return s.sample_walk(block, t, b, acc)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,empty", [(1, False), (5, False), (11, True), (12, False), (13, True), (16, False), (17, True),
                                     (20, True), (23, False)])
def test_indices_follow_the_rule(n, empty, precision):
    import ncsim_b200 as nb

    r = np.random.default_rng(n)
    v = r.normal(size=1 << n) + 1j * r.normal(size=1 << n)
    v *= r.random(1 << n) ** 3
    if empty:
        v[r.random(1 << n) < 0.3] = 0
        if n > 12:  # whole blocks without weight, the first and the last among them
            b = v.reshape(-1, 4096)
            b[0] = 0
            b[-1] = 0
            b[r.random(len(b)) < 0.3] = 0
            b[len(b) // 2, 77] = 1.0
    s = nb.GpuStateVector.from_amplitudes(v / np.linalg.norm(v), precision)
    u = np.concatenate([r.random(20000), [0.0, 1.0 - 2.0 ** -53, 0.5, 2.0 ** -60]])
    got = s.sample_uniforms(u)
    assert np.array_equal(got, _walked(s, n, u))
    assert np.all(np.abs(v[got.astype(np.int64)]) > 0)
