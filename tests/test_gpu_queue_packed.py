"""The tile queue of the packed length-gauge kernel, whose state between chunks holds
FP32 increments that are not folded yet: grids with more tiles than any occupancy of
the GPU holds (32 CTAs on each of its SMs), against launches of 64 steps, which are
not queued.  The same bits."""
import numpy as np
import pytest

import antelope_b200 as ab
from cases import variant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gauge,precision,rk,kpt", [("Wannier", "mixed", 4, 2), ("Wannier", "mixed", 5, 2),
                                                    ("Velocity", "fp64", 4, 1), ("Wannier", "fp64", 5, 1)])
def test_chunks_of_a_queued_launch(gauge, precision, rk, kpt):
    import torch
    points = (601, 600 * kpt // 2)
    assert points[0] * points[1] / (32 * kpt) > 32 * torch.cuda.get_device_properties(0).multi_processor_count
    c = variant(top__gauge=gauge, calc__Npoints=list(points), calc__RKorder=rk, calc__T1=250.0, pulse__ellip=0.3,
                pulse__ncycles=300.5 * 0.1 * 0.0855 / (2 * np.pi), calc__shotNumber=40)
    p = ab.Problem.from_dict(c)
    got = []
    for steps in (0, 64):   # 300 steps in chunks of 128, the last one partial
        s = ab.api.Solver(p, precision=precision, tile_k=32 * kpt, k_per_thread=kpt, steps_per_launch=steps)
        s.run()
        got.append((s.get(), s.snapshots()))
        s.close()
    (a, sa), (b, sb) = got
    for key in ("inter", "intra", "occ", "coh"):
        assert np.array_equal(getattr(a, key), getattr(b, key)), key
    for key in sa:
        assert np.array_equal(sa[key], sb[key]), key
