"""Three or more close bands in the plain method of the length gauge, against
the CPU oracle: clusters over the whole zone (from a tenth of the spectrum's
width down, partly filled), at one grid point only, and met by k + A(t) on the
way.  Bar: 1e-10 of max_t |J| (FP64 parity)."""
import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import wannier
from cases import variant
from oracle import pyoracle

pytestmark = pytest.mark.gpu


def _case(group, npoints, rk, steps=60.5, **calc):
    c = variant(top__gauge="Wannier", calc__Npoints=list(npoints), pulse__env_name="sin2", pulse__ellip=0.3,
                pulse__ncycles=steps * 0.1 * 0.0855 / (2 * np.pi))
    c["calc"].update(dict(rk=rk, tol=1e-8, T1=60.0, T2=40.0, **calc))
    del c["Haldane"]
    c["target"] = "SyntheticWannier"
    c["SyntheticWannier"] = group
    return c


def _group(nband, nval, h):
    """The seeded model's vectors and dipoles with other hoppings."""
    g = wannier.generate(50 + nband, nband=nband, nval=nval)
    g["h_re"] = [float(x) for x in h.real.reshape(-1)]
    g["h_im"] = [float(x) for x in h.imag.reshape(-1)]
    return g


def _frame(nband, nval):
    g = wannier.synthetic_model(wannier.generate(50 + nband, nband=nband, nval=nval))
    a = g["h"][0] + 1j * np.diag(np.arange(nband))
    return g["R"], np.linalg.qr(a + np.random.default_rng(nband).normal(size=a.shape))[0]


def _levels(nband, m):
    """Energies of the bands outside a cluster of m at 0: below, then above."""
    return np.array({1: [0.3], 2: [-0.3, 0.3], 3: [-0.3, 0.25, 0.5], 4: [-0.3, 0.2, 0.4, 0.6]}[nband - m])


def _cluster(nband, m, width):
    """m bands within about `width` of the spectrum's spread, half filled."""
    nval = nband // 2
    R, U = _frame(nband, nval)
    rows = np.r_[np.arange(m)]
    rest = np.arange(m, nband)
    small = wannier.synthetic_model(wannier.generate(70 + m, nband=m, nval=1, gap=0.0, h_scale=0.3 * width))["h"]
    other = wannier.synthetic_model(wannier.generate(80 + nband - m, nband=nband - m, nval=1, gap=0.0,
                                                     h_scale=0.01))["h"]
    h = np.zeros((len(R), nband, nband), complex)
    h[:, rows[:, None], rows] = small
    h[:, rest[:, None], rest] = other
    h[0, rest, rest] += _levels(nband, m)
    return _group(nband, nval, U @ h @ U.conj().T)


def _passing(nband, m, phi, closest):
    """A cluster of m bands whose width goes as closest + 1 - cos(k.a1 - phi)."""
    nval = nband // 2
    R, U = _frame(nband, nval)
    at = {tuple(r): i for i, r in enumerate(R)}
    rng = np.random.default_rng(m)
    c = rng.normal(size=(2, m, m)) + 1j * rng.normal(size=(2, m, m))
    c = 0.05 * (c + np.conj(np.swapaxes(c, 1, 2)))
    h = np.zeros((len(R), nband, nband), complex)
    width = {(0, 0): 1.0 + closest, (1, 0): -0.5 * np.exp(-1j * phi), (-1, 0): -0.5 * np.exp(1j * phi)}
    shape = {(0, 0): c[0], (0, 1): 0.2 * c[1], (0, -1): 0.2 * c[1]}   # C0 + 0.4 C1 cos(k.a2)
    for r1, w in width.items():
        for r2, x in shape.items():
            h[at[(r1[0] + r2[0], r1[1] + r2[1])], :m, :m] += w * x
    rest = np.arange(m, nband)
    h[at[(0, 0)], rest, rest] += _levels(nband, m)
    return _group(nband, nval, U @ h @ U.conj().T)


def _check(case):
    out, ref = ab.solve(case, precision="fp64"), pyoracle.run(case)
    scale = max(np.abs(ref["inter"]).max(), np.abs(ref["intra"]).max())
    err = max(np.abs(getattr(out, key) - ref[key]).max() for key in ("inter", "intra")) / scale
    assert err <= 1e-10, err
    N = ref["dims"]["nband"]
    assert np.abs(out.occ[:, :N] - ref["occ"]).max() < 1e-10
    return out


@pytest.mark.parametrize("nband,m", [(4, 3), (5, 3), (5, 4), (6, 3), (6, 4)])
@pytest.mark.parametrize("width", [1e-1, 1e-2, 1e-3, 1e-4])
def test_clusters_over_the_zone(nband, m, width):
    _check(_case(_cluster(nband, m, width), (4, 4), "rk4"))


@pytest.mark.parametrize("nband", [3, 4, 5, 6])
@pytest.mark.parametrize("width", [1e-2, 1e-4, 1e-6, 2e-7])
def test_close_pairs_over_the_zone(nband, width):
    """Two bands with gaps down to 2e-7 of the spectrum's width."""
    _check(_case(_cluster(nband, 2, width), (4, 4), "rk4"))


def _turn(c):
    """A_x where |A_x| is largest."""
    d = pyoracle.run(c)["dims"]
    A = np.array([pyoracle.laser_eval(c, d["atmin"] + c["calc"]["dt"] * n)[0][0] for n in range(d["Nt"])])
    return A[np.argmax(np.abs(A))]


def _strong(c, steps):
    """Linear field along a1 strong enough to carry k across the zone; a quarter of a cycle."""
    c["laser"]["pulses"][0].update(E0=0.05, ellip=0.0, ncycles=steps * 0.1 * 0.0855 / (2 * np.pi))
    return c


@pytest.mark.parametrize("nband,m", [(4, 3), (5, 3), (6, 3), (6, 4)])
@pytest.mark.parametrize("rk", ["rk4", "cashkarp45"])
@pytest.mark.parametrize("closest", [1e-2, 1e-3, 1e-4])
def test_cluster_met_on_the_way(nband, m, rk, closest):
    """Well separated bands at every grid point; k + A(t) enters the cluster
    where the field turns, and stays there for a while."""
    steps = 400.5
    c = _strong(_case(_passing(nband, m, 0.0, closest), (1, 13), rk), steps)
    turn = _turn(c) * 2.72
    assert abs(turn) > 0.2
    c = _strong(_case(_passing(nband, m, turn, closest), (1, 13), rk), steps)
    _check(c)


@pytest.mark.parametrize("nband,m", [(4, 3), (6, 4)])
def test_cluster_at_some_grid_points(nband, m):
    """Grids of which one or a few rows of points lie in the cluster, a batch of
    them with a model without one: the batch equals the solves alone."""
    # k.a1 = 2 pi f0 on the grid's rows f0 = -1/2 ... 1/2: the cluster is at f0 = 0
    cases = [_case(_passing(nband, m, 0.0, 1e-4), n, "rk4", steps=s) for n, s in (((31, 3), 20.5), ((100, 101), 3.5))]
    cases.append(_case(wannier.generate(9, nband=nband, nval=nband // 2), (5, 7), "rk4", steps=30.5))
    outs = [_check(c) for c in cases]
    b = ab.Batch([ab.Problem.from_dict(c) for c in cases], precision="fp64")
    b.run()
    for i, one in enumerate(outs):
        for key in ("inter", "intra", "occ"):
            np.testing.assert_array_equal(getattr(b.get(i), key), getattr(one, key))
    b.close()


@pytest.mark.parametrize("rk", [4, 5])
@pytest.mark.parametrize("closest", [1e-3, 1e-4, 1e-5])
@pytest.mark.parametrize("E0", [0.0, 4e-5, 0.0045])
def test_four_band_material(rk, closest, E0):
    """Two Haldane layers whose bottom Dirac cone (mass `closest`) touches the
    top layer's upper band at K; K is reached where the field turns (E0 = 0: a
    weak one that stays in the cone)."""
    phi0, t2, top = 1.16, 0.025, 0.06
    K = 4 * np.pi / (3 * np.sqrt(3) * 1.44 / 0.52917721067)
    f3 = 2 * np.sin(phi0)
    # at K: sum cos(k.b) = -3/2, sum sin(k.b) = -3 sqrt(3) / 2
    sins = sum(np.sin(K * x) for x in (np.sqrt(3) * 1.44 / 0.52917721067,) + (-np.sqrt(3) / 2 * 1.44 / 0.52917721067,) * 2)
    t2b = t2 - top / (1.5 * 2 * np.cos(phi0))
    c = variant(top__gauge="Wannier", calc__RKorder=rk, calc__T1=25.0, calc__T2=10.0, calc__Npoints=[1, 3],
                pulse__E0=E0 or 0.2 * closest,
                calc__BZaxes=[0.01, 0.0, 0.0, 0.0, 8 * closest, 0.0, 0.0, 0.0, 0.0], calc__BZorigin=[0.0, 0.0])
    del c["Haldane"]
    c["target"] = "Haldane2L"
    c["Haldane2L"] = {"t1": 0.075, "t2": t2, "phi0": phi0, "a0": 1.44, "t11": closest, "polytype": "AB",
                      "M0": float(top + f3 * t2 * sins), "t2_bottom": float(t2b),
                      "M0_bottom": float(f3 * t2b * top + closest)}
    c["calc"]["BZorigin"] = [float(K - _turn(c)), 0.0]
    _check(c)
