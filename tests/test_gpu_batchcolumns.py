"""Laser columns that a batch evaluates ahead: every get, repeated and from several
threads at once, returns the solve's own."""
import threading

import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 2, 5])
def test_gets_in_any_order_and_again(threads):
    probs = [ab.Problem.from_dict(c) for c in workloads.scan_cases(n=24, precision="mixed")]
    b = ab.Batch(probs, precision="mixed")
    b.run()
    got = [[None, None] for _ in probs]

    def work(k):
        for rep in range(2):
            for i in range(k, len(probs), threads):
                got[len(probs) - 1 - i][rep] = b.get(len(probs) - 1 - i)
    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    b.close()
    for p, (x, y) in zip(probs, got):
        assert np.array_equal(x.laser, p.laser())
        for key in ("inter", "intra", "occ", "coh", "laser"):
            assert np.array_equal(getattr(x, key), getattr(y, key)), key
