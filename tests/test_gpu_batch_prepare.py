"""GPU test of how Batch.prepare() plans its circuits."""
import os
import time

import pytest

from nqpu_b200 import circuits
from nqpu_b200.batch import Batch
from nqpu_b200.state import Circuit

pytestmark = pytest.mark.gpu


@pytest.mark.skipif(len(os.sched_getaffinity(0)) < 16, reason="fewer than 16 host cores")
def test_plans_on_many_host_threads():
    # 256 circuits on the sixteen threads that 16 of them each allow: more than four
    # times as fast as one after the other, which four threads could not be
    items = [(Circuit(n, g), J, h) for n, g, J, h in circuits.hea_batch(256, 1, nmin=10, nmax=20)]
    serial, plans = [], []
    for _ in range(10):
        t = time.perf_counter()
        for c, _J, h in items:
            c.plan_stats(len(h), "c64", "tiled")
        serial.append(time.perf_counter() - t)
        b = Batch()
        for c, J, h in items:
            b.add_ising(c, J, h)
        b.prepare()
        plans.append(b.stats()["prepare_s"]["plans"])
        b.close()
    assert min(serial) >= 4.2 * min(plans)
