"""The many-steps-per-launch kernels of fixed-step N-band solves against the
CPU oracle, at grids around their block sizes and step counts around their
launch length.  Bar: 1e-10 of max_t |J| per current series (FP64 parity)."""
import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import wannier
from cases import material, variant
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _table(nband, gauge, npoints, rk, steps, **calc):
    c = variant(top__gauge=gauge, calc__Npoints=list(npoints), calc__RKorder=rk, pulse__env_name="sin2",
                pulse__ellip=0.3, pulse__ncycles=steps * 0.1 * 0.0855 / (2 * np.pi))
    c["calc"].update(calc)
    del c["Haldane"]
    c["target"] = "SyntheticWannier"
    c["SyntheticWannier"] = wannier.generate(3 + nband, nband=nband, nval=nband // 2)
    return c


def _check(case):
    out, ref = ab.solve(case, precision="fp64"), pyoracle.run(case)
    scale = max(np.abs(ref["inter"]).max(), np.abs(ref["intra"]).max())
    for key in ("inter", "intra"):
        assert np.abs(getattr(out, key) - ref[key]).max() <= 1e-10 * scale, key
    N = ref["dims"]["nband"]
    assert np.abs(out.occ[:, :N] - ref["occ"]).max() < 1e-10
    return out


@pytest.mark.parametrize("nband", [2, 3, 4, 5, 6, 8])
@pytest.mark.parametrize("rk", [4, 5])
@pytest.mark.parametrize("npoints,steps", [((1, 1), 1.5), ((7, 9), 64.5), ((8, 8), 63.5), ((5, 13), 130.5)])
def test_velocity_gauge_matches_oracle(nband, rk, npoints, steps):
    _check(_table(nband, "Velocity", npoints, rk, steps, T1=250.0))


# Grids without a point where bands meet (even point counts): there the
# dephasing depends on the basis inside the pair, i.e. on rounding.
@pytest.mark.parametrize("name", ["WilsonMass", "TMDCs", "KaneMele", "Haldane2L"])
@pytest.mark.parametrize("rk", [4, 5])
@pytest.mark.parametrize("npoints,steps", [((2, 1), 63.5), ((4, 8), 64.5), ((6, 11), 130.5)])
def test_material_length_gauge_matches_oracle(name, rk, npoints, steps):
    c = material(name, "Wannier", calc__T1=250.0, calc__RKorder=rk, pulse__ellip=0.3,
                 pulse__ncycles=steps * 0.1 * 0.0855 / (2 * np.pi))
    c["calc"]["Npoints"] = list(npoints)
    _check(c)


def test_batch_and_snapshots_equal_the_solve_alone():
    """Different lengths, grids and band counts in one batch, with snapshots
    (which end launches early) and without: bitwise the solves alone."""
    cases = [_table(4, "Velocity", (7, 10), 4, 150.5), _table(4, "Velocity", (9, 9), 4, 70.5, shotNumber=20),
             _table(2, "Velocity", (3, 5), 5, 100.5), material("TMDCs", "Velocity", calc__shotNumber=3),
             material("KaneMele", "Wannier", calc__shotNumber=3), material("KaneMele", "Wannier", calc__RKorder=5)]
    probs = [ab.Problem.from_dict(c) for c in cases]
    b = ab.Batch(probs, precision="fp64", use_graph=True)
    b.run()
    for i, p in enumerate(probs):
        s = ab.api.Solver(p, precision="fp64")
        s.run()
        alone, got = s.get(), b.get(i)
        for key in ("inter", "intra", "occ", "coh"):
            assert np.array_equal(getattr(alone, key), getattr(got, key)), (i, key)
        assert s.steps() == b.steps(i)
        if "shotNumber" in cases[i]["calc"]:
            x, y = s.snapshots(), b.snapshots(i)
            assert all(np.array_equal(x[key], y[key]) for key in x), i
        s.close()
    b.close()
