"""Performance cases of the propagator: what its users run, from the smallest
call to the largest, through the package's public entry points.

A case is a dict of plain values; ``prepare`` turns it into parsed problems
(what a program has in hand after reading its inputParam.cfg files), ``run``
makes one pass -- a whole solve, batch or burst of requests, with its output
arrays on the host -- and ``exact`` integrates the same equations with plain
torch in 64 bits where that is quick.

Mixed-precision Haldane cases name their launch shape (tile_k, k_per_thread),
as a program does that wants its numbers to the last bit from run to run: the
autotuner picks a shape by timing, and the FP32 part of the k-sum depends on
it.  The FP64 cases leave the shape to the autotuner, as a plain call does.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from antelope_b200 import wannier
from antelope_b200.workloads import haldane_case, omega_of_um, scan_cases, serving_cases

BOHR_ANG = 0.529177210903
W0_32UM = 0.014238          # 3.2 um
W0_SHORT = 0.0855           # the tests' short-wavelength pulse


# ------------------------------------------------------------------ the cases
def _case(name, kind="solve", **kw):
    c = {"name": name, "kind": kind, "model": "Haldane", "gauge": "Velocity", "precision": "fp64", "rk": "rk4",
         "n0": 8, "n1": 10, "w0": W0_SHORT, "ncycles": 2.0, "env": "cos4", "T1": -1.0, "T2": 220.0,
         "inter_intra": True, "shots": 0, "hmax": 0, "tile_k": 0, "count": 1, "shapes": 1, "graph": False, "nband": 6}
    c.update(kw)
    return c


def listed():
    return [
        # a convergence or unit check of a new input file: tens of k-points, one
        # short pulse; nothing but latency (the tests' own size)
        _case("smallest"),
        # the plain method's configuration: 150 x 150, 8 cycles at 3.2 um
        _case("plain_150", n0=150, n1=150, w0=W0_32UM, ncycles=8.0, env="sin2"),
        # the converged grid of the same solve in both methods
        _case("plain_600", n0=600, n1=600, w0=W0_32UM, ncycles=8.0, env="sin2"),
        _case("mixed_600", n0=600, n1=600, w0=W0_32UM, ncycles=8.0, env="sin2", precision="mixed", tile_k=512),
        # the reference's defaults -- length gauge, RKorder 5, total current only
        # -- with T1, on an odd grid, with density snapshots
        _case("length_default", gauge="Wannier", rk="rk5", n0=240, n1=251, w0=W0_32UM, ncycles=2.0, T1=300.0,
              inter_intra=False, shots=2),
        # the length gauge in the mixed method, with the spectrum taken on the GPU
        _case("length_mixed", gauge="Wannier", n0=400, n1=401, w0=W0_32UM, ncycles=4.0, env="sin2",
              precision="mixed", tile_k=256, hmax=30),
        # a slice of the (M/t2, phi0, ellipticity) scan: uneven grids and pulses
        # in one batch, the time loop as a CUDA graph
        _case("scan", kind="scan", precision="mixed", tile_k=512, count=10, graph=True),
        # a burst of one-colour and two-colour requests to the resident server
        _case("serve", kind="serve", precision="mixed", tile_k=512, count=12),
        # N = 6 Wannier tables with dipoles, adaptive Cash-Karp, length gauge
        _case("wannier6", model="SyntheticWannier", gauge="Wannier", rk="cashkarp45", n0=100, n1=100, w0=W0_32UM,
              ncycles=0.25, env="sin2"),
        # several seeds of it as one mixed-precision batch
        _case("wannier6_batch", kind="wannier_batch", model="SyntheticWannier", gauge="Wannier", rk="cashkarp45",
              n0=48, n1=49, w0=W0_32UM, ncycles=0.125, env="sin2", precision="mixed", count=4, graph=True),
        # an analytic four-band material in the velocity gauge
        _case("kanemele_velocity", model="KaneMele", n0=120, n1=121, T1=300.0),
        # a three-band transition-metal dichalcogenide with the reference's
        # defaults (length gauge, RKorder 5)
        _case("tmdc_length", model="TMDCs", gauge="Wannier", rk="rk5", n0=48, n1=50),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _cycles(w0, steps):
    """Pulse cycles whose duration is about `steps` steps of dt = 0.1."""
    return round(max(0.05, steps * 0.1 * w0 / (2 * math.pi)), 3)


def draw(rng):
    """One more case: single solves of every model family, both gauges and
    methods, and small scans, over the range the listed cases span."""
    fam = rng.choice(["haldane"] * 4 + ["material"] * 3 + ["wannier"] * 2 + ["scan"])
    gauge = rng.choice(["Velocity", "Wannier"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    T1 = rng.choice([-1.0, -1.0, 300.0])
    env = rng.choice(["cos4", "sin2"])
    if fam == "scan":
        c = _case("", kind="scan", precision="mixed", tile_k=512, count=rng.randint(2, 8),
                  shapes=rng.randrange(1 << 20), graph=rng.random() < 0.5)
    elif fam == "haldane":
        n0, n1 = int(_log(rng, 6, 600)), int(_log(rng, 6, 600))
        w0 = round(omega_of_um(_log(rng, 0.533, 3.2)), 6)
        steps = min(_log(rng, 800, 35000), 1.0e10 / (n0 * n1))
        c = _case("", gauge=gauge, precision=precision, rk=rng.choice(["rk4", "rk4", "rk5"]), n0=n0, n1=n1, w0=w0,
                  ncycles=_cycles(w0, steps), env=env, T1=T1, inter_intra=rng.random() < 0.7,
                  hmax=rng.choice([0, 0, 15]))
        if precision == "mixed":
            c["tile_k"] = 512 if n0 * n1 >= 100000 else 128
    elif fam == "material":
        model = rng.choice(["KaneMele", "WilsonMass", "TMDCs", "Haldane2L"])
        n0, n1 = int(_log(rng, 4, 120)), int(_log(rng, 4, 120))
        steps = min(_log(rng, 300, 1500), 5.0e6 / (n0 * n1))
        c = _case("", model=model, gauge=gauge, precision=precision, rk=rng.choice(["rk4", "rk5"]), n0=n0, n1=n1,
                  ncycles=_cycles(W0_SHORT, max(steps, 100)), env=env, T1=T1)
    else:
        n0, n1 = int(_log(rng, 4, 100)), int(_log(rng, 4, 100))
        steps = min(_log(rng, 300, 1100), 5.0e6 / (n0 * n1))
        c = _case("", model="SyntheticWannier", gauge=gauge, precision=precision, n0=n0, n1=n1, w0=0.057,
                  rk=rng.choice(["rk4", "rk5", "cashkarp45", "cashkarp45"]), nband=rng.choice([3, 4, 6, 6]),
                  ncycles=_cycles(0.057, max(steps, 100)), env=env, T1=T1)
    del c["name"]
    return c


# ------------------------------------------------------------ inputs of a case
def _config(case, seed, i=0):
    """The inputParam.cfg (dict form) of a single solve: laser and model
    parameters drawn from the seed."""
    rng = np.random.default_rng([seed, i])
    c = haldane_case()
    c["gauge"] = case["gauge"]
    p = c["laser"]["pulses"][0]
    p.update(E0=float(rng.uniform(0.002, 0.006)), w0=float(case["w0"]), ncycles=float(case["ncycles"]),
             env_name=case["env"], ellip=float(rng.choice([0.0, 0.25, 0.5])), cep=float(rng.uniform(0.0, 360.0)),
             phix=float(rng.uniform(0.0, 60.0)))
    k = c["calc"]
    k.update(Npoints=[int(case["n0"]), int(case["n1"])], T1=float(case["T1"]), T2=float(case["T2"]),
             InterIntra=bool(case["inter_intra"]), precision=case["precision"], rk=case["rk"], tol=1e-8)
    if case["shots"]:
        k["shotNumber"] = int(case["shots"])
    model = case["model"]
    mt2, phi0 = float(rng.uniform(1.0, 4.0)), float(rng.uniform(0.6, 1.5))
    if model == "Haldane":
        c["Haldane"].update(Mt2=mt2, phi0=phi0)
        return c
    del c["Haldane"]
    c["target"] = model
    if model == "SyntheticWannier":
        n = int(case["nband"])
        c[model] = wannier.generate(int(rng.integers(1 << 30)), nband=n, nval=n // 2)
    elif model == "KaneMele":
        c[model] = {"t1": 0.075, "t2": 0.025, "tR": float(rng.uniform(0.005, 0.02)), "Mt2": mt2, "phi0": phi0,
                    "a0": 1.44}
    elif model == "WilsonMass":
        c[model] = {"t": 0.02, "delta": float(rng.uniform(0.01, 0.02)), "mu": -0.03, "a0": 5.0, "a1": 6.0}
    elif model == "Haldane2L":
        c[model] = {"t1": 0.075, "t2": 0.025, "phi0": phi0, "a0": 1.44, "t11": float(rng.uniform(0.005, 0.02)),
                    "polytype": "AB", "Mt2": mt2}
    else:
        c[model] = {"Material": str(rng.choice(["MoS2", "WS2", "MoSe2", "WSe2"]))}
    return c


def _configs(case, seed):
    """The cfgs of a pass.  A scan or a request stream keeps the grids and the
    pulse lengths of the case's own number `shapes`; its material, ellipticity,
    phases and field strengths follow the seed."""
    n = int(case["count"])
    if case["kind"] not in ("scan", "serve"):
        return [_config(case, seed, i) for i in range(n)]
    if case["kind"] == "scan":
        gen = lambda s: scan_cases(n, seed=s, precision=case["precision"])  # noqa: E731
    else:
        gen = lambda s: serving_cases(n, seed=s, precision=case["precision"])[1]  # noqa: E731
    rng = np.random.default_rng(seed)
    out = gen(int(case["shapes"]))
    for c, other in zip(out, gen(seed)):
        c["Haldane"] = other["Haldane"]
        for p in c["laser"]["pulses"]:
            p.update(cep=float(rng.uniform(0.0, 360.0)), ellip=other["laser"]["pulses"][0]["ellip"],
                     E0=p["E0"] * float(rng.uniform(0.8, 1.2)))
    return out


def _opts(case):
    o = {"precision": case["precision"]}
    if case["tile_k"]:
        o.update(tile_k=int(case["tile_k"]), k_per_thread=2)
    return o


def prepare(case, seed):
    import antelope_b200 as ab
    state = {"case": case, "problems": [ab.Problem.from_dict(c) for c in _configs(case, seed)]}
    if case["kind"] == "serve":   # the resident server a program keeps
        state["server"] = ab.Server(**_opts(case))
    return state


def _arrays(out, laser=True):
    d = {"inter": out.inter, "intra": out.intra, "occ": out.occ, "coh": out.coh}
    if laser:
        d["laser"] = out.laser
    return d


def run(state):
    from antelope_b200.api import Batch, Solver
    case, probs = state["case"], state["problems"]
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit(p) for p in probs]
        return [_arrays(srv.wait(i)[0]) for i in ids]
    if case["kind"] != "solve":
        b = Batch(probs, use_graph=bool(case["graph"]), **_opts(case))
        try:
            b.run()
            if case["kind"] == "scan":
                return [dict(_arrays(b.get(i)), harmonics=b.harmonics(i, W0_32UM, 25)) for i in range(len(probs))]
            return [_arrays(b.get(i)) for i in range(len(probs))]
        finally:
            b.close()
    s = Solver(probs[0], **_opts(case))
    try:
        s.run()
        out = _arrays(s.get())
        if case["shots"]:
            out["snapshots"] = s.snapshots()
        if case["hmax"]:
            out["harmonics"] = s.harmonics(float(case["w0"]), int(case["hmax"]))
        return out
    finally:
        s.close()


# --------------------------------------------------------------- work of a pass
_STAGES = {"rk4": 4, "rk5": 6, "cashkarp45": 6}
_BANDS = {"Haldane": 2, "KaneMele": 4, "WilsonMass": 2, "TMDCs": 3, "Haldane2L": 4}


def _steps(cfg):
    """Output times of a solve: pulses centred on t0 with cos4 / sin2
    envelopes, dt steps over the longest."""
    half = max(p["ncycles"] * math.pi / p["w0"] for p in cfg["laser"]["pulses"])
    return max(1, int(math.floor(2 * half / cfg["calc"]["dt"])))


def work(case):
    """Operations: per k-point and stage the commutator of Hermitian N x N
    matrices (8 N^3), H (velocity gauge 4 N^2; length gauge 8 N^2 per lattice
    vector pair) and the stage sums (6 N^2); in the length gauge also the basis
    change of the dephasing (16 N^3).  Two bands: the Hermitian-minimal count
    (198 per RK4 step in the velocity gauge, 364 in the length gauge; 1.87
    times that for six stages).  Bytes: the output arrays and the tables."""
    flops = nbytes = 0.0
    for cfg in _configs(case, 1):
        n, nt = cfg["calc"]["Npoints"][0] * cfg["calc"]["Npoints"][1], _steps(cfg)
        N = int(case["nband"]) if case["model"] == "SyntheticWannier" else _BANDS[case["model"]]
        S, vg = _STAGES[case["rk"]], cfg["gauge"] == "Velocity"
        if case["model"] in ("Haldane", "WilsonMass"):
            per = (198.0 if vg else 364.0) * (1.0 if S == 4 else 1.87)
        else:
            pairs = 19 if case["model"] == "SyntheticWannier" else 7
            per = S * (8.0 * N ** 3 + 6.0 * N * N + (4.0 * N * N if vg else 8.0 * N * N * pairs + 16.0 * N ** 3))
        flops += per * n * nt
        nbytes += 8.0 * nt * (3 + 3 + N + 1 + 2 + 7)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------ 64-bit comparison
def _laser(cfg):
    """A(t), E(t) of the pulses and the time grid (t_min, dt, Nt)."""
    ps = cfg["laser"]["pulses"]
    dt = cfg["calc"]["dt"]

    def raw(t):
        A, E = np.zeros(t.shape + (3,)), np.zeros(t.shape + (3,))
        for p in ps:
            w, n, th = p["w0"], p["ncycles"], math.radians(p["cep"])
            half, ef = n * math.pi / w, w / (2 * n)
            k = t - p["t0"]
            q = 4 if p["env_name"] == "cos4" else 2
            on = np.abs(k) <= half
            f = np.where(on, np.cos(k * ef) ** q, 0.0)
            fp = np.where(on, -q * ef * np.sin(k * ef) * np.cos(k * ef) ** (q - 1), 0.0)
            s, c = np.sin(k * w - th), np.cos(k * w - th)
            g = math.sqrt(1.0 / (1.0 + p["ellip"] ** 2))
            ex, ey = g * p["E0"], g * p["E0"] * p["ellip"]
            px = math.radians(p["phix"])
            ux, uy = np.array([math.cos(px), math.sin(px), 0.0]), np.array([-math.sin(px), math.cos(px), 0.0])
            A += (-ex / w * s * f)[..., None] * ux + (ey / w * c * f)[..., None] * uy
            E += (ex * c * f - ex / w * s * fp)[..., None] * ux + (ey * s * f + ey / w * c * fp)[..., None] * uy
        return A, E

    half = max(p["ncycles"] * math.pi / p["w0"] for p in ps)
    t0 = -half
    A0, E0 = raw(np.array(t0))
    return (lambda t: tuple(x - y for x, y in zip(raw(np.asarray(t)), (A0, E0)))), t0, dt, int(math.floor(2 * half / dt))


def _honeycomb(a):
    r3 = math.sqrt(3.0)
    return (a * np.array([[0.0, 1.0], [-r3 / 2, -0.5], [r3 / 2, -0.5]]),
            a * np.array([[r3, 0.0], [-r3 / 2, 1.5], [-r3 / 2, -1.5]]))


def _haldane_block(k, m, phi, va, vb):
    """(H, -dH/dk) of a Haldane layer at the points k."""
    t1, t2 = m["t1"], m["t2"]
    a, b = k @ va.T, k @ vb.T
    b0 = 2 * t2 * math.cos(phi) * np.cos(b).sum(1)
    b3 = m["Mt2"] * t2 - 2 * t2 * math.sin(phi) * np.sin(b).sum(1)
    off = t1 * np.exp(-1j * a).sum(1)
    H = np.stack([b0 + b3, off, off.conj(), b0 - b3], 1).reshape(-1, 2, 2).astype(complex)
    J = []
    for x in range(2):
        d0 = -2 * t2 * math.cos(phi) * (np.sin(b) @ vb[:, x])
        d3 = -2 * t2 * math.sin(phi) * (np.cos(b) @ vb[:, x])
        do = t1 * (np.exp(-1j * a) @ (-1j * va[:, x]))
        J.append(-np.stack([d0 + d3, do, do.conj(), d0 - d3], 1).reshape(-1, 2, 2))
    return H, J


def _model(cfg):
    """(H and J at points k, Brillouin-zone axes, occupied bands)."""
    name, m = cfg["target"], cfg[cfg["target"]]
    if name == "SyntheticWannier":
        t = wannier.synthetic_model(m)
        L = np.array(t["lattice"]).reshape(2, 2)
        R = t["R"] @ L

        def hj(k):
            ph = np.exp(1j * k @ R.T)
            H = np.einsum("kr,rij->kij", ph, t["h"])
            J = []
            for x in range(2):
                D = np.einsum("kr,rij->kij", ph, t["d"][:, x])
                dH = np.einsum("kr,rij->kij", ph * (1j * R[:, x]), t["h"])
                J.append(-dH + 1j * (D @ H - H @ D))
            return H, J
        return hj, 2 * math.pi * np.linalg.inv(L).T, t["nval"]
    if name == "WilsonMass":
        a0, a1, t, d = m["a0"], m["a1"], m["t"], m["delta"]

        def hj(k):
            x, y = a0 * k[:, 0], a1 * k[:, 1]
            mat = lambda b1, b2, b3: np.stack([b3, b1 - 1j * b2, b1 + 1j * b2, -b3], 1).reshape(-1, 2, 2)  # noqa: E731
            z = np.zeros(len(k))
            return (mat(d * np.sin(x), d * np.sin(y), -2 * t * (np.cos(x) + np.cos(y)) - m["mu"]),
                    [-mat(a0 * d * np.cos(x), z, 2 * t * a0 * np.sin(x)),
                     -mat(z, a1 * d * np.cos(y), 2 * t * a1 * np.sin(y))])
        return hj, np.diag([2 * math.pi / a0, 2 * math.pi / a1]), 1
    if name in ("Haldane", "KaneMele"):
        a = m["a0"] / BOHR_ANG
        va, vb = _honeycomb(a)
        axes = np.diag([2 * math.pi / math.sqrt(3.0) / a, 4 * math.pi / 3.0 / a])
        if name == "Haldane":
            return (lambda k: _haldane_block(k, m, m["phi0"], va, vb)), axes, 1
        cR = np.array([1.0, np.exp(2j * math.pi / 3), np.exp(-2j * math.pi / 3)])

        def hj(k):
            up, dn = _haldane_block(k, m, m["phi0"], va, vb), _haldane_block(k, m, -m["phi0"], va, vb)
            e = np.exp(1j * k @ va.T)
            H = np.zeros((len(k), 4, 4), complex)
            H[:, :2, :2], H[:, 2:, 2:] = up[0], dn[0]
            r = 1j * m["tR"]
            H[:, 0, 3] = r * (e @ cR.conj())
            H[:, 1, 2] = r * (e.conj() @ cR.conj())
            H[:, 2, 1], H[:, 3, 0] = H[:, 1, 2].conj(), H[:, 0, 3].conj()
            J = []
            for x in range(2):
                g = np.zeros((len(k), 4, 4), complex)
                g[:, :2, :2], g[:, 2:, 2:] = up[1][x], dn[1][x]
                # the model's own current operator: the Rashba entries carry +dH/dk,
                # its (3, 0) entry without the factor i tR
                iv = 1j * va[:, x]
                g[:, 0, 3] = r * (e @ (cR.conj() * iv))
                g[:, 1, 2] = r * (e.conj() @ (cR.conj() * -iv))
                g[:, 2, 1] = -r * (e @ (cR * iv))
                g[:, 3, 0] = -(e.conj() @ (cR * -iv))
                J.append(g)
            return H, J
        return hj, axes, 2
    return None


_TABLEAU = {
    "rk4": ([0, 0.5, 0.5, 1.0], [[], [0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 2 / 6, 2 / 6, 1 / 6]),
    "rk5": ([0, 0.25, 3 / 8, 12 / 13, 1.0, 0.5],
            [[], [1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
             [439 / 216, -8.0, 3680 / 513, -845 / 4104], [-8 / 27, 2.0, -3544 / 2565, 1859 / 4104, -11 / 40]],
            [16 / 135, 0.0, 6656 / 12825, 28561 / 56430, -9 / 50, 2 / 55]),
}


def exact(case, seed):
    """The output arrays of a single fixed-step solve from plain torch in 64
    bits: every model written out above in the velocity gauge, the two-band
    ones in the length gauge too (its dephasing needs the instantaneous
    eigenbasis, closed-form for two bands).  None for batches and servers, for
    adaptive steps, for other models and for solves of over about 20 s."""
    if case["kind"] != "solve" or case["rk"] not in _TABLEAU:
        return None
    cfg = _config(case, seed)
    vg, got = cfg["gauge"] == "Velocity", _model(cfg)
    cs, aij, bs = _TABLEAU[case["rk"]]
    nk, nt = case["n0"] * case["n1"], _steps(cfg)
    if got is None or nt * len(cs) > 60000 or nk * nt * len(cs) > 6.0e8:
        return None
    hj, axes, nval = got
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    up = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)  # noqa: E731
    field, t0, dt, Nt = _laser(cfg)
    grid = [np.arange(n) / (n - 1) - 0.5 if n > 1 else np.zeros(1) for n in (case["n0"], case["n1"])]
    wt = [np.where((np.arange(n) == 0) | (np.arange(n) == n - 1), 0.5, 1.0) if n > 1 else np.ones(1)
          for n in (case["n0"], case["n1"])]
    f = np.stack(np.meshgrid(*grid, indexing="ij"), -1).reshape(-1, 2)
    k, w = f @ axes, np.outer(*wt).reshape(-1)
    H, J = hj(k)
    N = H.shape[1]
    if not vg and N != 2:
        return None
    dV = abs(np.linalg.det(axes)) / nk
    t = t0 + dt * np.arange(Nt)
    A, E = field(t)
    As = np.stack([A] + [field(t + c * dt)[0] for c in cs[1:]], 1)      # [Nt][stage][3]
    g1 = 1.0 / case["T1"] if case["T1"] > 0 else 0.0
    g2 = 1.0 / case["T2"] if case["T2"] > 0 else 0.0
    eps, U = np.linalg.eigh(H)
    occ0 = (np.arange(N) < nval).astype(float)
    wd = up(w)
    eye = torch.eye(N, dtype=torch.complex128, device=dev)
    if vg:
        P = [up(np.conj(np.swapaxes(U, 1, 2)) @ j @ U) for j in J]
        e, rho0 = torch.diag_embed(up(eps)).to(torch.complex128), torch.diag(up(occ0)).to(torch.complex128)
        rho = rho0.expand(nk, N, N).clone()
        G = g2 * (1 - eye.real) + g1 * eye.real

        def rhs(y, a):
            HY = (e + float(a[0]) * P[0] + float(a[1]) * P[1]) @ y
            return -1j * (HY - HY.mH) - G * (y - rho0)

        def currents(y, a):
            tot = [torch.einsum("k,kij,kji->", wd + 0j, y, p).real for p in P]
            ia = [torch.einsum("k,ki,ki->", wd + 0j, y.diagonal(dim1=1, dim2=2), p.diagonal(dim1=1, dim2=2)).real
                  for p in P]
            return [tot[x] - ia[x] for x in range(2)] + ia
    else:
        # the model as Fourier data of k: re-evaluated at k + A by its own formulas
        rho = up(np.einsum("kim,m,kjm->kij", U, occ0, U.conj()))
        hjt = _two_band_torch(cfg, up(k), dev)

        def split(a, current):
            """(H, unit vector projector pair difference S = n.sigma, J) at k + A."""
            h, j = hjt(float(a[0]), float(a[1]), current)
            tr = 0.5 * (h[:, 0, 0] + h[:, 1, 1])
            h0 = h - tr[:, None, None] * eye
            bn = torch.sqrt((h0[:, 0, 0] * h0[:, 0, 0].conj() + h0[:, 0, 1] * h0[:, 0, 1].conj()).real)
            return h, h0 / torch.clamp(bn, min=1e-300)[:, None, None], j

        def rhs(y, a):
            h, s, _ = split(a, False)
            HY = h @ y
            d = 0.5 * (y + s @ y @ s)          # the band-diagonal part of rho
            return -1j * (HY - HY.mH) - g1 * d - g2 * (y - d)

        def currents(y, a):
            _, s, j = split(a, True)
            d = 0.5 * (y + s @ y @ s)
            tot = [torch.einsum("k,kij,kji->", wd + 0j, y, q).real for q in j]
            ia = [torch.einsum("k,kij,kji->", wd + 0j, d, q).real for q in j]
            return [tot[x] - ia[x] for x in range(2)] + ia

    sums = torch.zeros((Nt, 4), dtype=torch.float64, device=dev)
    dens = torch.zeros((Nt, N, N), dtype=torch.complex128, device=dev)
    for n in range(Nt):
        sums[n] = torch.stack(currents(rho, As[n, 0]))
        dens[n] = torch.einsum("k,kij->ij", wd + 0j, rho)
        ks = []
        for i in range(len(cs)):
            y = rho
            for a, q in zip(aij[i], ks):
                if a:
                    y = y + dt * a * q
            ks.append(rhs(y, As[n, i]))
        rho = rho + sum(dt * b * q for b, q in zip(bs, ks) if b)
    sums, dens = sums.cpu().numpy(), dens.cpu().numpy()
    inter, intra = np.zeros((Nt, 3)), np.zeros((Nt, 3))
    inter[:, :2], intra[:, :2] = sums[:, :2], sums[:, 2:]
    if vg:
        intra += nval * A * w.sum()
    if not case["inter_intra"]:
        inter, intra = inter + intra, np.zeros((Nt, 3))
    occ = np.real(np.einsum("nii->ni", dens)) / nk
    out = {"inter": inter * dV, "intra": intra * dV, "occ": np.concatenate([occ, occ.sum(1, keepdims=True)], 1),
           "coh": None, "laser": np.concatenate([t[:, None], E, A], 1)}
    el = nval * N + nval + 1
    if not vg or N == 2:   # in the band basis of more bands it depends on the eigenvectors' phases
        flat = np.concatenate([dens.reshape(-1), np.zeros(N * N)]) / nk
        z = flat[np.arange(Nt) * N * N + el]
        out["coh"] = np.stack([z.real, z.imag], 1)
    return out


def _two_band_torch(cfg, k, dev):
    """H and J of the two-band models at k + A on the device."""
    m = cfg[cfg["target"]]
    mat = lambda b0, b1, b2, b3: torch.stack([b0 + b3 + 0j, b1 - 1j * b2, b1 + 1j * b2, b0 - b3 + 0j],  # noqa: E731
                                             1).reshape(-1, 2, 2)
    if cfg["target"] == "WilsonMass":
        a0, a1, t, d = m["a0"], m["a1"], m["t"], m["delta"]

        def hj(ax, ay, current):
            x, y = a0 * (k[:, 0] + ax), a1 * (k[:, 1] + ay)
            z = torch.zeros_like(x)
            h = mat(z, d * torch.sin(x), d * torch.sin(y), -2 * t * (torch.cos(x) + torch.cos(y)) - m["mu"])
            j = [-mat(z, a0 * d * torch.cos(x), z, 2 * t * a0 * torch.sin(x)),
                 -mat(z, z, a1 * d * torch.cos(y), 2 * t * a1 * torch.sin(y))] if current else None
            return h, j
        return hj
    va, vb = (torch.as_tensor(v, device=dev) for v in _honeycomb(m["a0"] / BOHR_ANG))
    t1, t2, phi = m["t1"], m["t2"], m["phi0"]
    c2, s2 = 2 * t2 * math.cos(phi), 2 * t2 * math.sin(phi)

    def hj(ax, ay, current):
        q = k + torch.tensor([ax, ay], dtype=torch.float64, device=dev)
        a, b = q @ va.T, q @ vb.T
        ca, sa, cb, sb = torch.cos(a), torch.sin(a), torch.cos(b), torch.sin(b)
        h = mat(c2 * cb.sum(1), t1 * ca.sum(1), t1 * sa.sum(1), m["Mt2"] * t2 - s2 * sb.sum(1))
        j = [-mat(-c2 * (sb @ vb[:, x]), -t1 * (sa @ va[:, x]), t1 * (ca @ va[:, x]), -s2 * (cb @ vb[:, x]))
             for x in range(2)] if current else None
        return h, j
    return hj
