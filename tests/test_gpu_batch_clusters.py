"""Trajectories shared by a cluster of CTAs: a few trajectories (clusters of 8, 4 or 2)
give the bits that the same trajectories give among many (one CTA each), for
registers of one tile up to 64, both kernel forms, records with and without
outcomes above the tile's qubits, and batches of one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(nb, count, seed0, n_lo, n_span, depth, cfg):
    b = nb.TrajectoryBatch.random_layers(count, seed0=seed0, n_lo=n_lo, n_span=n_span, depth=depth, p=0.02)
    try:
        for n in range(n_lo, n_lo + n_span):  # the same plan whatever the autotuner would pick
            b.set_knob_set(n, 0, final=n == n_lo + n_span - 1)
    except nb.SimError:
        pass  # knobs already final from the cache: the same for both batches
    b.set_config(**cfg)
    b.run()
    return b.results()


@pytest.mark.parametrize("cfg", [dict(ctas_per_sm=1, buffers=2), dict(ctas_per_sm=2, buffers=1), dict(ctas_per_sm=1, buffers=1)])
@pytest.mark.parametrize("n_lo,n_span,few", [(13, 1, 3), (14, 3, 5), (17, 3, 1), (16, 4, 40)])
def test_few_equal_many(n_lo, n_span, few, cfg):
    import ncsim_b200 as nb

    alone = _batch(nb, few, 77, n_lo, n_span, 8, cfg)
    among = _batch(nb, 700, 77, n_lo, n_span, 8, cfg)
    for x, y in zip(alone, among):
        assert np.array_equal(x, y[:few])


def test_given_circuits_with_few_measurements():
    import ncsim_b200 as nb

    n = 17
    base = nb.Circuit.random_layers(n, 6, 3, 0.05, 0, 0).to_text()
    for m in (0, 1, 5, 13, 14, 17):
        text = base + "".join(f"M {q}\n" for q in range(m))
        one = nb.TrajectoryBatch.from_circuits([nb.Circuit.parse(text)], [5])
        one.set_config(ctas_per_sm=1, buffers=2)
        one.run()
        many = nb.TrajectoryBatch.from_circuits([nb.Circuit.parse(text)] * 400, [5] + list(range(100, 499)))
        many.set_config(ctas_per_sm=1, buffers=2)
        many.run()
        for x, y in zip(one.results(), many.results()):
            assert np.array_equal(x, y[:1])
