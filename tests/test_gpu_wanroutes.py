"""Which N-band solves the many-step and projection kernels take, and how."""
import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import wannier
from cases import variant
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _table(nband, npoints, rk="rk4", steps=40.5, gauge="Wannier", **calc):
    c = variant(top__gauge=gauge, calc__Npoints=list(npoints), pulse__env_name="sin2", pulse__ellip=0.3,
                pulse__ncycles=steps * 0.1 * 0.0855 / (2 * np.pi))
    c["calc"].update(dict(rk=rk, tol=1e-8, T1=250.0, **calc))
    del c["Haldane"]
    c["target"] = "SyntheticWannier"
    c["SyntheticWannier"] = wannier.generate(30 + nband, nband=nband, nval=nband // 2)
    return c


def _axes(a=2.72):
    b = 2 * np.pi * np.linalg.inv(wannier.lattice_vectors(a)).T
    return np.array([[b[0, 0], b[0, 1], 0.0], [b[1, 0], b[1, 1], 0.0], [0.0, 0.0, 0.0]])


@pytest.mark.parametrize("tilt", [1e-10, 1e-12])
def test_axes_of_ten_digits(tilt):
    """A zone axis that leaves vectors b.R apart by less than a user's digits:
    they share no phase along a row.  Bar: 1e-10 of max_t |J|."""
    axes = _axes()
    axes[1, 0] += tilt
    axes[1, 1] -= tilt
    c = _table(6, (3, 8), steps=200.5, BZaxes=[float(x) for x in axes.reshape(-1)])
    out, ref = ab.solve(c, precision="fp64"), pyoracle.run(c)
    scale = max(np.abs(ref["inter"]).max(), np.abs(ref["intra"]).max())
    for key in ("inter", "intra"):
        assert np.abs(getattr(out, key) - ref[key]).max() <= 1e-10 * scale, key
