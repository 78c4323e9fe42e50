"""A batch's run leaves the caller to itself while the GPU works, and get, from
one thread or several, gives each solve's own columns."""
import threading
import time

import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import workloads

pytestmark = pytest.mark.gpu


def test_run_returns_before_the_gpu_and_gets_agree():
    import torch
    probs = [ab.Problem.from_dict(c) for c in workloads.scan_cases(n=64, precision="mixed")]
    outs = {}
    for threads in (1, 4):
        b = ab.Batch(probs, precision="mixed", use_graph=True, steps_per_launch=256)
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        t = time.perf_counter()
        b.run(stream.cuda_stream)
        queued = time.perf_counter() - t
        if threads == 1:
            stream.synchronize()
            total = time.perf_counter() - t
            assert queued < 0.8 * total, (queued, total)
            got = [b.get(i) for i in range(len(probs))]
        else:
            got = [None] * len(probs)

            def work(k):
                for i in range(k, len(probs), threads):
                    got[i] = b.get(i)
            ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
            [x.start() for x in ts]
            [x.join() for x in ts]
        outs[threads] = got
        b.close()
    for p, x, y in zip(probs, outs[1], outs[4]):
        for key in ("inter", "intra", "occ", "coh", "laser"):
            assert np.array_equal(getattr(x, key), getattr(y, key)), key
        assert x.laser.shape[0] == p.dims.Nt
