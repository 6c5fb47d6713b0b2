"""The cluster sizes that a batch takes, by its device time: 148 trajectories of one size fill the
SMs with one CTA each and take as long as one trajectory on one CTA; 74, 37 and 18 of them share
the same SMs in clusters of 2, 4 and 8.  Also a sample timed by `tune` runs in the clusters of the
whole batch, whatever the sample's own size."""
from __future__ import annotations

import time

import pytest

pytestmark = pytest.mark.gpu

N, DEPTH = 18, 40  # 32 tiles


def _batch(nb, count, cfg):
    b = nb.TrajectoryBatch.random_layers(count, seed0=5, n_lo=N, n_span=1, depth=DEPTH, p=0.01)
    try:
        b.set_knob_set(N, 0, final=True)
    except nb.SimError:
        pass
    if cfg:
        b.set_config(**cfg)
    return b


@pytest.mark.parametrize("cfg", [dict(ctas_per_sm=1, buffers=2), dict(ctas_per_sm=1, buffers=1)])
def test_smaller_batches_share_the_sms_in_clusters(cfg):
    import ncsim_b200 as nb

    sms = nb.device_info()["sm_count"]
    ms = {}
    for count in (sms, sms // 2, sms // 4, sms // 8, 1):
        b = _batch(nb, count, cfg)
        ms[count] = min(b.run() for _ in range(4))
    # a cluster of C takes 1 / C of the tiles and a fixed part per pass; without clusters all are equal
    assert ms[sms // 2] < 0.8 * ms[sms]
    assert ms[sms // 4] < 0.55 * ms[sms]
    assert ms[sms // 8] < 0.4 * ms[sms] and ms[1] < 0.4 * ms[sms]


def test_a_sample_is_timed_in_the_batchs_clusters():
    import ncsim_b200 as nb

    sms = nb.device_info()["sm_count"]
    b = _batch(nb, 4 * sms, None)  # so many take one CTA each
    b.tune(sms // 8)
    t = time.perf_counter()
    b.tune(sms // 8)  # four configurations, twice each
    took = 1e3 * (time.perf_counter() - t)
    one = _batch(nb, sms, dict(ctas_per_sm=1, buffers=2))
    ms = min(one.run() for _ in range(3))
    # on one CTA each run takes as long as one trajectory does; in clusters of 8 a quarter
    assert took > 5 * ms, (took, ms)
