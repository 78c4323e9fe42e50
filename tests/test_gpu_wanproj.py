"""The projection attempt kernel (explicit tables, length gauge, FP64) against
the CPU oracle: band counts, step rules, grids at the edges of its blocks and
rows, and with and without dipoles.  Bar: 1e-10 of max_t |J| (FP64 parity)."""
import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import wannier
from cases import variant
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _case(nband, npoints, rk, steps=40.5, dipoles=True, **calc):
    c = variant(top__gauge="Wannier", calc__Npoints=list(npoints), pulse__env_name="sin2", pulse__ellip=0.3,
                pulse__ncycles=steps * 0.1 * 0.0855 / (2 * np.pi))
    c["calc"].update(dict(rk=rk, tol=1e-8, T1=250.0, **calc))
    del c["Haldane"]
    c["target"] = "SyntheticWannier"
    g = wannier.generate(20 + nband, nband=nband, nval=nband // 2)
    if not dipoles:
        del g["d_re"], g["d_im"]
    c["SyntheticWannier"] = g
    return c


def _check(case):
    out, ref = ab.solve(case, precision="fp64"), pyoracle.run(case)
    scale = max(np.abs(ref["inter"]).max(), np.abs(ref["intra"]).max())
    for key in ("inter", "intra"):
        assert np.abs(getattr(out, key) - ref[key]).max() <= 1e-10 * scale, key
    N = ref["dims"]["nband"]
    assert np.abs(out.occ[:, :N] - ref["occ"]).max() < 1e-10


@pytest.mark.parametrize("nband", [3, 4, 5, 6])
@pytest.mark.parametrize("rk", ["rk4", "rk5", "cashkarp45"])
@pytest.mark.parametrize("npoints", [(6, 5), (1, 9), (9, 1), (3, 2)])
def test_matches_oracle(nband, rk, npoints):
    _check(_case(nband, npoints, rk))


@pytest.mark.parametrize("npoints,calc", [((6, 5), dict(ksfactor=[0.5, 0.8, 1.0])),
                                          ((5, 6), dict(BZaxes=[1.2, 0.1, 0.0, -0.2, 0.9, 0.0, 0.0, 0.0, 0.0],
                                                        BZorigin=[0.05, -0.1]))])
def test_other_zones_and_no_dipoles(npoints, calc):
    _check(_case(6, npoints, "rk4", **calc))
    _check(_case(4, npoints, "cashkarp45", dipoles=False, **calc))


def test_slices_add_up():
    p = ab.Problem.from_dict(_case(6, (7, 5), "rk4"))
    total = 0.0
    for a, b in ((0, 11), (11, 12), (12, 35)):   # slices that start and end inside a row
        s = ab.api.Solver(p, k_slice=(a, b), precision="fp64")
        s.run()
        total = total + s.sums()
        s.close()
    out, whole = ab.api.assemble(p, total), ab.solve(p, precision="fp64")
    for key in ("inter", "intra", "occ"):
        x, y = getattr(out, key), getattr(whole, key)
        assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max(), key


@pytest.mark.parametrize("nband,npoints", [(3, (1, 10)), (3, (3, 7)), (4, (1, 16)), (4, (17, 1)), (5, (1, 6)), (5, (1, 7)),
                                           (6, (1, 10)), (6, (11, 1)), (6, (2, 5)), (6, (7, 3))])
def test_edges_of_a_block(nband, npoints):
    """A block's k-points (32 lanes in whole groups): full, one more, and rows that end inside it."""
    _check(_case(nband, npoints, "cashkarp45"))


def test_batch_of_step_rules_equals_the_solves_alone():
    """Solves of one launch differ in their stages, grids and lengths."""
    cases = [_case(6, (3, 7), "rk4", steps=20.5), _case(6, (5, 5), "cashkarp45"), _case(6, (1, 11), "rk5", steps=12.5),
             _case(4, (3, 7), "cashkarp45"), _case(4, (1, 17), "rk4")]
    problems = [ab.Problem.from_dict(c) for c in cases]
    b = ab.Batch(problems, precision="fp64")
    b.run()
    outs = [b.get(i) for i in range(len(cases))]
    b.close()
    for p, out in zip(problems, outs):
        one = ab.solve(p, precision="fp64")
        for key in ("inter", "intra", "occ"):
            np.testing.assert_array_equal(getattr(out, key), getattr(one, key))
