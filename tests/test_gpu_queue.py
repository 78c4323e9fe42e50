"""Launches whose tiles outnumber the CTAs the GPU holds run through the tile
queue (chunks of steps handed to the resident CTAs).  The same tiles in
launches of 64 steps, which are not queued, give the same bits."""
import numpy as np
import pytest

import antelope_b200 as ab
from cases import variant

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gauge,precision,rk,kpt", [("Velocity", "fp64", 4, 1), ("Velocity", "fp64", 5, 2),
                                                    ("Wannier", "fp64", 4, 1), ("Wannier", "fp64", 5, 1),
                                                    ("Wannier", "mixed", 4, 2), ("Wannier", "mixed", 5, 2)])
@pytest.mark.parametrize("npoints", [(281, 280), (401, 333)])
def test_queued_launches_give_the_same_bits(gauge, precision, rk, kpt, npoints):
    # 300 steps: chunks of 128 steps in the default launches of 1024, the last
    # one partial; 32-thread CTAs, so that thousands of tiles are needed
    c = variant(top__gauge=gauge, calc__Npoints=list(npoints), calc__RKorder=rk, calc__T1=250.0, pulse__ellip=0.3,
                pulse__ncycles=300.5 * 0.1 * 0.0855 / (2 * np.pi), calc__shotNumber=40)
    p = ab.Problem.from_dict(c)
    got = []
    for steps in (0, 64):
        s = ab.api.Solver(p, precision=precision, tile_k=32 * kpt, k_per_thread=kpt, steps_per_launch=steps)
        s.run()
        got.append((s.get(), s.snapshots()))
        s.close()
    (a, sa), (b, sb) = got
    for key in ("inter", "intra", "occ", "coh"):
        assert np.array_equal(getattr(a, key), getattr(b, key)), key
    for key in sa:
        assert np.array_equal(sa[key], sb[key]), key
