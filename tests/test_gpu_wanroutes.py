"""Which N-band solves the many-step and projection kernels take, and what the
server's admission counts for them."""
import numpy as np
import pytest

import antelope_b200 as ab
from antelope_b200 import api, wannier
from cases import material, variant
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


def _equal(out, one):
    for key in ("inter", "intra", "occ"):
        np.testing.assert_array_equal(getattr(out, key), getattr(one, key))


def _base_bytes(p, nR):
    """Device memory of a solve on the attempt kernels alone."""
    N, nk, Nt = p.dims.nband, p.dims.ntotal, p.dims.Nt
    return 4 * nk * N * N * 16 + nk * 8 + nR * N * N * 80 + nR * 16 + nR * 3456 + nk // 4 * 136 + Nt * 128 + (1 << 20)


def _served(p, budget):
    srv = ab.Server(precision="fp64", mem_budget_bytes=float(budget))
    try:
        return srv.wait(srv.submit(p), timeout=120.0)[0]
    finally:
        srv.close()


def _close(out, one, tol=1e-12):
    scale = max(np.abs(one.inter).max(), np.abs(one.intra).max())
    for key in ("inter", "intra"):
        assert np.abs(getattr(out, key) - getattr(one, key)).max() <= tol * scale, key


def test_admission_of_long_and_thin_grids():
    """No row tables for a material, and none above their limit."""
    km = material("KaneMele", "Wannier", pulse__ncycles=0.05)
    km["calc"]["Npoints"] = [4000, 1]
    for c, nR in ((_table(6, (1200, 1), rk="cashkarp45", steps=3.5), 37), (km, 19)):
        p = ab.Problem.from_dict(c)
        out = _served(p, _base_bytes(p, nR))
        assert np.abs(out.intra).max() > 0.0


@pytest.mark.parametrize("gauge", ["Velocity", "Wannier"])
def test_a_budget_without_room_for_tables(gauge):
    """The solve runs on the kernels that need none: no less is admitted than they hold."""
    c = _table(6, (64, 60), steps=10.5, gauge=gauge)
    p = ab.Problem.from_dict(c)
    nk = p.dims.ntotal
    budget = _base_bytes(p, 37) + (nk * 6 * 16 + nk * 3 * 36 * 16 if gauge == "Velocity" else 0)
    _close(_served(p, budget), ab.solve(p, precision="fp64"), 1e-11)


def test_a_finished_request_is_noticed():
    """A request alone on the server: its 10 steps are one tick (32 attempts, 64
    launches), and the server sees it done a few ticks later."""
    p = ab.Problem.from_dict(_table(6, (64, 60), steps=10.5))
    for _ in range(3):
        srv = ab.Server(precision="fp64")
        srv.wait(srv.submit(p), timeout=120.0)
        launches = srv.stats()["launches"]
        srv.close()
        assert launches <= 20 * 64, launches


def test_row_tables_above_their_limit():
    """A grid of very many short rows runs on the tracked kernel; its slices, whose
    tables fit, on the projections.  Bar: 1e-10 of max_t |J| (FP64 parity)."""
    n = (50000, 2)   # 24 kB of tables a row: 1.2 GB
    p = ab.Problem.from_dict(_table(6, n, steps=6.5))
    total = 0.0
    for a in range(0, 100000, 25000):
        s = api.Solver(p, k_slice=(a, a + 25000), precision="fp64")
        s.run()
        total = total + s.sums()
        s.close()
    _close(api.assemble(p, total), ab.solve(p, precision="fp64"), 1e-10)


@pytest.mark.parametrize("shots", [1, 400])
def test_snapshots_do_not_slow_the_server(shots):
    """A request returns the output files' arrays: beside a long two-band solve
    (one turn of the server per tick of it) the turns it takes do not depend on
    its snapshot count."""
    long = variant(calc__Npoints=[200, 200], pulse__ncycles=60000.5 * 0.1 * 0.0855 / (2 * np.pi))
    launches, outs = [], []
    for n in (0, shots):
        c = _table(4, (6, 5), steps=300.5, gauge="Velocity", shotNumber=n)
        srv = ab.Server(precision="fp64", steps_per_launch=64)
        other = srv.submit(ab.Problem.from_dict(long))
        while srv.stats()["launches"] < 4:
            pass
        before = srv.stats()["launches"]
        out, _ = srv.wait(srv.submit(ab.Problem.from_dict(c)), timeout=120.0)
        launches.append(srv.stats()["launches"] - before)
        srv.cancel(other)
        srv.close()
        outs.append(out)
    _equal(outs[1], outs[0])
    assert launches[1] <= 3 * launches[0], launches


@pytest.mark.parametrize("shots", [200, 700])
def test_snapshots_do_not_idle_a_batch(shots):
    """Launches end at snapshots: a batch queues as many between two looks at its
    controllers as 64 steps take.  A short solve with snapshots beside a long
    adaptive one, whose attempts every look costs 64 of."""
    c = _table(4, (6, 5), steps=600.5, gauge="Velocity", shotNumber=shots)
    other = _table(3, (4, 4), rk="cashkarp45", steps=10.5)
    n = []
    for cases in ([other], [c, other]):
        b = ab.Batch([ab.Problem.from_dict(x) for x in cases], precision="fp64")
        b.run()
        n.append(b.launches)
        b.close()
    # 600 steps are 10 looks: 128 launches of the other class each, and at most 3 per step
    assert n[1] <= 12 * 128 + 3 * 700, n


def test_requests_that_join_and_leave():
    """Plain length-gauge, velocity-gauge and two-band requests come in while
    others run; some are cancelled at once.  Each result is the solve's alone."""
    cases = [_table(6, (7, 5)), _table(6, (5, 9), rk="cashkarp45", steps=25.5), _table(3, (4, 4), rk="rk5"),
             material("KaneMele", "Wannier"), material("TMDCs", "Wannier", calc__RKorder=5),
             _table(5, (9, 3), gauge="Velocity"), variant(calc__Npoints=[40, 41]), _table(4, (1, 17), steps=90.5)]
    probs = [ab.Problem.from_dict(c) for c in cases]
    alone = [ab.solve(p, precision="fp64") for p in probs]
    srv = ab.Server(precision="fp64")
    ids, dropped = [], []
    for rep in range(3):
        for i, p in enumerate(probs):
            ids.append((i, srv.submit(p)))
            if (i + rep) % 3 == 0:
                dropped.append(srv.submit(p))
                srv.cancel(dropped[-1])
        if rep == 1:
            out, _ = srv.wait(ids[0][1], timeout=120.0)
            _equal(out, alone[0])
            ids.pop(0)
    for i, rid in ids:
        out, _ = srv.wait(rid, timeout=120.0)
        if cases[i]["target"] == "Haldane":   # the server's CTA sizes: other sums over k
            for key in ("inter", "intra"):
                x, y = getattr(out, key), getattr(alone[i], key)
                assert np.abs(x - y).max() <= 1e-12 * np.abs(y).max()
        else:
            _equal(out, alone[i])
    srv.close()
