"""Performance cases: the work that users of this engine have it do, through its Python entry points.

Kinds of case (the "kind" of a case dict):
  solve   one grid, one operating point: new injections go up, gbpf_solve runs the Newton loop, and the state, flows,
          switch events and history come back (what the command-line driver and an interactive study do)
  batch   many load scenarios of one or several grids in one launch: arrays up, solve, per-bus results down
  warm    the same on one grid, started from a network's prediction
  train   epochs of training of that network, then its weights

Grids are the committed inputs of the tests and the benchmark, or seeded generator grids of other sizes.  Loads and
generation are drawn around the file's values, close enough that Newton converges for every scenario.
"""
import functools
import gzip
import importlib
import math
import os
import tempfile

import numpy as np
import torch

gb = importlib.import_module("experience-of-using-gpu-in-power-flow-computation_gb300")
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")

IEEE = {14: "ieee14", 30: "ieee30", 57: "ieee57", 118: "ieee118", 236: "ieee118x2", 472: "ieee118x4",
        944: "ieee118x8", 1888: "ieee118x16", 3776: "ieee118x32", 7552: "ieee118x64"}
MIXED = ("c4_14", "c4_30", "c4_57", "c4_118", "c4_236", "c4_472")


# ------------------------------------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: one operating point of a textbook grid, limits on (latency and launches)
        {"name": "solve_14_fp64_limits", "kind": "solve", "grid": "ieee14", "precision": "fp64", "limits": True,
         "dense": False},
        # the usual single study: 118 buses, reactive limits
        {"name": "solve_118_fp64_limits", "kind": "solve", "grid": "ieee118", "precision": "fp64", "limits": True,
         "dense": False},
        # a regional grid, one operating point
        {"name": "solve_1888_fp64", "kind": "solve", "grid": "c5_base", "precision": "fp64", "limits": False,
         "dense": False},
        # an interconnection, one operating point, limits on
        {"name": "solve_15104_fp64_limits", "kind": "solve", "grid": "c3_base", "precision": "fp64", "limits": True,
         "dense": False},
        # a large grid with the FP32 factorisation
        {"name": "solve_7552_fp32", "kind": "solve", "grid": "ieee118x64", "precision": "fp32", "limits": False,
         "dense": False},
        # the reference's dense method (metodo = denso) on a grid where its cubic work is felt
        {"name": "solve_944_dense", "kind": "solve", "grid": "ieee118x8", "precision": "fp64", "limits": False,
         "dense": True},
        # a day of load scenarios of the 118-bus grid
        {"name": "batch_118_fp32", "kind": "batch", "grid": "c2_base", "precision": "fp32", "limits": False,
         "n": 4096},
        # a contingency-study-sized batch in full precision with limits, an odd count
        {"name": "batch_118_fp64_limits", "kind": "batch", "grid": "c2_base", "precision": "fp64", "limits": True,
         "n": 999},
        # scenarios of the regional grid, one thread block each
        {"name": "batch_1888_fp32", "kind": "batch", "grid": "c5_base", "precision": "fp32", "limits": False,
         "n": 2048},
        # grids of uneven size in one launch
        {"name": "batch_mixed_fp32", "kind": "batch", "grid": "mixed", "precision": "fp32", "limits": False,
         "n": 1500},
        # the learned start, serving: features, network, start choice, Newton
        {"name": "warm_1888_fp32", "kind": "warm", "grid": "c5_base", "precision": "fp32", "limits": False,
         "n": 2048},
        # training of that network
        {"name": "train_1888", "kind": "train", "grid": "c5_base", "width": 512, "layers": 3, "rows": 4096,
         "batch": 1024, "epochs": 24, "metric": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "dense", "batch", "batch", "batch", "mixed", "warm", "train"])
    if kind in ("solve", "dense"):
        top = 944 if kind == "dense" else 15104
        want = _log_int(rng, 14, top)
        if want <= 472 and rng.random() < 0.5:
            grid = "gen_%d_%d" % (want, rng.randrange(1, 1000))  # any size, odd ones among them
        elif want > 10000:
            grid = "c3_base"
        else:
            grid = IEEE[min(IEEE, key=lambda n: abs(math.log(n / want)))]
        fp32 = kind == "solve" and rng.random() < 0.4
        small = grid in ("ieee14", "ieee30", "ieee57", "ieee118")
        return {"kind": "solve", "grid": grid, "precision": "fp32" if fp32 else "fp64",
                "limits": bool(small and not fp32 and kind == "solve" and rng.random() < 0.5),
                "dense": kind == "dense"}
    if kind == "batch":
        big = rng.random() < 0.35
        fp32 = rng.random() < 0.6
        if big:
            return {"kind": "batch", "grid": "c5_base", "precision": "fp32" if fp32 else "fp64", "limits": False,
                    "n": _log_int(rng, 1, 2048 if fp32 else 1000)}
        grid = rng.choice(["ieee14", "ieee57", "ieee118", "c2_base", "c2_base", "c4_236", "gen"])
        if grid == "gen":
            grid = "gen_%d_%d" % (_log_int(rng, 14, 300), rng.randrange(1, 1000))
        return {"kind": "batch", "grid": grid, "precision": "fp32" if fp32 else "fp64",
                "limits": bool(not fp32 and grid in ("ieee14", "ieee118", "c2_base") and rng.random() < 0.4),
                "n": _log_int(rng, 1, 4096 if fp32 else 1500)}
    if kind == "mixed":
        return {"kind": "batch", "grid": "mixed", "precision": rng.choice(["fp32", "fp64"]), "limits": False,
                "n": _log_int(rng, 16, 1500)}
    if kind == "warm":
        return {"kind": "warm", "grid": rng.choice(["ieee118", "c2_base", "ieee118x8", "c5_base"]),
                "precision": rng.choice(["fp32", "fp32", "fp64"]), "limits": False, "n": _log_int(rng, 33, 2048)}
    return {"kind": "train", "grid": rng.choice(["ieee118", "c4_236", "ieee118x8", "c5_base"]),
            "width": rng.choice([128, 256, 512]), "layers": rng.choice([2, 3]), "rows": 8 * _log_int(rng, 128, 512),
            "batch": rng.choice([256, 512, 1000, 1024]), "epochs": rng.randrange(2, 9),
            "metric": rng.random() < 0.5}


# ------------------------------------------------------------------------------------------------- grids
@functools.lru_cache(maxsize=None)
def grid_of(name):
    if name.startswith("gen_"):
        _, nbus, seed = name.split("_")
        return gb.generate(4, int(seed), nbus=int(nbus))
    for sub, ext in (("", ".cdf"), ("", ".cdf.gz"), ("", ".cdfx.gz"), ("ieee", ".cdf.gz")):
        src = os.path.join(GOLDEN, sub, name + ext)
        if os.path.exists(src):
            break
    if not src.endswith(".gz"):
        return gb.read_grid(src)
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, name + ext[:-3])
        with gzip.open(src, "rb") as f, open(path, "wb") as o:
            o.write(f.read())
        return gb.read_grid(path)


def _names(case):
    return MIXED if case["grid"] == "mixed" else (case["grid"],)


# Load spread of the scenarios (sigma of the lognormal factor) and half width of the generation factors: half of what
# the benchmark draws on its 118-bus grid, where one scenario in a thousand has no solution that Newton finds
SPREAD = 0.05


def _scenarios(name, n, rng):
    b = grid_of(name).buses()
    sl = sg = SPREAD
    nb = len(b["Pload"])
    lf = np.exp(rng.normal(-0.5 * sl * sl, sl, (n, nb)))
    return b["Pload"] * lf, b["Qload"] * lf, b["Pg"] * rng.uniform(1 - sg, 1 + sg, (n, nb))


def inputs(case, seed):
    """Host arrays of one pass: grid index per instance and the packed loads and active generation."""
    rng = np.random.default_rng(seed)
    names = _names(case)
    n = case.get("n", 1)
    gi = rng.permutation(n).astype(np.int32) % len(names)  # as many of each grid, in any order
    per = {t: [a for a in zip(*_scenarios(names[t], int((gi == t).sum()), rng))] for t in range(len(names))}
    at = dict.fromkeys(per, 0)
    rows = []
    for t in gi:
        rows.append(per[t][at[t]])
        at[t] += 1
    return gi, [np.concatenate([r[q] for r in rows]) for q in range(3)]


def _tol(case):
    """The benchmark's 1e-8; two decades further with the FP32 factorisation on the larger grids, so that the answer is
    a converged one and not the FP32 rounding of the last step."""
    large = case["grid"] != "mixed" and grid_of(case["grid"]).nB > 500
    return 1e-10 if case["precision"] == "fp32" and large else 1e-8


def _options(case):
    return dict(tolerancia=_tol(case), no_max_iter=100, lim_inj_reat=int(case["limits"]),
                metodo=int(case.get("dense", False)),
                precision=gb.PREC_FP32_IR if case["precision"] == "fp32" else gb.PREC_FP64)


# ------------------------------------------------------------------------------- plain 64-bit power flow (no engine)
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class Net:
    """One grid's arrays and dense Ybus in 64 bits."""

    def __init__(self, name):
        g = grid_of(name)
        b, br, pv = g.buses(), g.branches(), g.pvpq()
        n, dev = g.nB, _device()
        self.n, self.dev = n, dev
        f, t = br["from_bus"] - 1, br["to_bus"] - 1
        y = 1.0 / (br["r"] + 1j * br["x"])
        tap = br["tap_re"] + 1j * br["tap_im"]
        self.Y = torch.zeros((n, n), dtype=torch.complex128, device=dev)

        def add(i, j, v):
            self.Y.index_put_((torch.as_tensor(i, device=dev).long(), torch.as_tensor(j, device=dev).long()),
                              torch.as_tensor(v, device=dev), accumulate=True)

        add(f, t, -y / np.conj(tap))
        add(t, f, -y / tap)
        add(f, f, y / np.abs(tap) ** 2 + 0.5j * br["bch"])
        add(t, t, y + 0.5j * br["bch"])
        add(np.arange(n), np.arange(n), b["gsh"] + 1j * b["bsh"])
        self.type, self.base = b["type"], b
        self.ns = np.where(b["type"] != 3)[0]
        self.pq = np.where(b["type"] <= 1)[0]
        self.pv, self.Qmin, self.Qmax = pv["pv"] - 1, pv["Qmin"], pv["Qmax"]
        self.f, self.t, self.br = f, t, br
        nz = torch.nonzero(self.Y)
        self.Ys = torch.sparse_coo_tensor(nz.T, self.Y[nz[:, 0], nz[:, 1]], (n, n)).to_sparse_csr()

    def injections(self, V, th):
        """[S, n] magnitudes and angles -> complex power."""
        u = torch.polar(V, th)
        return u * torch.conj((self.Ys @ u.T.contiguous()).T)

    def jacobian(self, V, th):
        """d[P; Q] / d[theta; V] of one state, [2n, 2n]."""
        u = torch.polar(V, th)
        e = torch.polar(torch.ones_like(V), th)
        I = self.Y @ u
        dth = 1j * u[:, None] * torch.conj(torch.diag(I) - self.Y * u[None, :])
        dV = u[:, None] * torch.conj(self.Y * e[None, :]) + torch.diag(torch.conj(I) * e)
        return torch.cat([torch.cat([dth.real, dV.real], 1), torch.cat([dth.imag, dV.imag], 1)], 0)

    def chord(self, P, Q):
        """Solutions of the scenarios [S, n] without limits: Newton on their mean, then chord steps for all."""
        dev, n = self.dev, self.n
        at = torch.as_tensor(np.concatenate([self.ns, n + self.pq]), device=dev)
        V0 = torch.as_tensor(self.base["V0"], device=dev)
        t0 = torch.as_tensor(self.base["theta0"], device=dev)
        P, Q = torch.as_tensor(P, device=dev), torch.as_tensor(Q, device=dev)

        def step(V, th, lu, p, q):
            s = self.injections(V, th)
            g = torch.cat([p - s.real, q - s.imag], 1)[:, at]
            dx = torch.linalg.lu_solve(*lu, g.T.contiguous()).T
            x = torch.cat([th, V], 1)
            x[:, at] += dx
            return x[:, n:].contiguous(), x[:, :n].contiguous(), float(g.abs().max())

        Vm, tm = V0[None].clone(), t0[None].clone()
        pm, qm = P.mean(0, keepdim=True), Q.mean(0, keepdim=True)
        for k in range(2 if n > 4000 else 5):
            lu = torch.linalg.lu_factor(self.jacobian(Vm[0], tm[0])[at][:, at])
            for _ in range(1 if n <= 4000 or k == 0 else 2):
                Vm, tm, g = step(Vm, tm, lu, pm, qm)
            if g < 1e-9:
                break
        V, th = Vm.repeat(len(P), 1), tm.repeat(len(P), 1)
        best = math.inf
        for k in range(200):
            V1, t1, g = step(V, th, lu, P, Q)
            if not g < best and k > 4 and best < 1e-9:
                break
            V, th, best = V1, t1, min(best, g)
        return V, th

    def newton(self, P, Q, Qload, tol, max_iter=100):
        """The scenarios [S, n] by full Newton with the PV <-> PQ rules, all of them together (small grids)."""
        dev, n, S = self.dev, self.n, len(P)
        T = lambda a: torch.as_tensor(np.array(a), device=dev)  # noqa: E731
        P, Q, Qload = T(P), T(Q).clone(), T(Qload)
        V, th = T(self.base["V0"]).repeat(S, 1), T(self.base["theta0"]).repeat(S, 1)
        act = T((self.type <= 1)).repeat(S, 1)
        ns, pv = T(self.ns), T(self.pv)
        qmin, qmax = T(self.Qmin), T(self.Qmax)
        dxm = torch.full((S,), math.inf, dtype=torch.float64, device=dev)
        done = torch.zeros(S, dtype=torch.bool, device=dev)
        more = 3  # steps past the engine's test, to rounding, the limits left as they are
        for it in range(max_iter):
            s = self.injections(V, th)
            if it >= 1 and len(pv):
                go = ((dxm < 10 * tol) & ~done)[:, None]
                qg = s.imag[:, pv] + Qload[:, pv]
                lo, hi = qg < qmin - tol, qg > qmax + tol
                at = act[:, pv]
                new = torch.where(lo, qmin - Qload[:, pv], torch.where(hi, qmax - Qload[:, pv], Q[:, pv]))
                Q[:, pv] = torch.where(go & (lo | hi), new, Q[:, pv])
                act[:, pv] = torch.where(go, lo | hi, at)
            gp = (P - s.real)[:, ns]
            gq = torch.where(act, Q - s.imag, torch.zeros_like(V))[:, ns]
            g = torch.cat([gp, gq], 1)
            done |= g.abs().amax(1) <= tol
            more -= bool(done.all())
            if not more:
                break
            u, e = torch.polar(V, th), torch.polar(torch.ones_like(V), th)
            I = (self.Y @ u.T).T
            yu = self.Y[None] * u[:, None, :]
            dth = 1j * u[:, :, None] * torch.conj(torch.diag_embed(I) - yu)
            dV = u[:, :, None] * torch.conj(self.Y[None] * e[:, None, :]) + torch.diag_embed(torch.conj(I) * e)
            a = act[:, ns]
            J = torch.zeros((S, 2 * len(ns), 2 * len(ns)), dtype=torch.float64, device=dev)
            m = len(ns)
            J[:, :m, :m] = dth.real[:, ns][:, :, ns]
            J[:, :m, m:] = dV.real[:, ns][:, :, ns] * a[:, None, :]
            J[:, m:, :m] = dth.imag[:, ns][:, :, ns] * a[:, :, None]
            J[:, m:, m:] = torch.where(a[:, :, None] & a[:, None, :], dV.imag[:, ns][:, :, ns],
                                       torch.eye(m, dtype=torch.float64, device=dev) * (~a)[:, None, :])
            dx = torch.linalg.solve(J, g)
            th[:, ns] += dx[:, :m]
            V[:, ns] += dx[:, m:]
            dxm = dx.abs().amax(1)
        return V, th

    def flows(self, V, th):
        """Branch flows of one state as GPU/PQcalc.cuh:523-557 defines them."""
        V, th, Y = V.cpu().numpy(), th.cpu().numpy(), self.Y.cpu().numpy()
        br, first, ph = self.br, {}, {}
        for i, (a, b) in enumerate(zip(self.f, self.t)):
            first.setdefault((min(a, b), max(a, b)), i)
            ph.setdefault((a, b), br["phase"][i])
        bsh = np.array([br["bch"][first[(min(a, b), max(a, b))]] for a, b in zip(self.f, self.t)])
        phi = np.array([ph[(a, b)] for a, b in zip(self.f, self.t)])
        k, m = self.f, self.t
        ang = phi + th[k] - th[m]
        ca, sa, ykm, ymk = np.cos(ang), np.sin(ang), Y[k, m], Y[m, k]
        vv = V[k] * V[m]
        return {"Pdp": V[k] ** 2 * ykm.real - vv * ykm.real * ca - vv * ykm.imag * sa,
                "Ppd": V[m] ** 2 * ymk.real - vv * ymk.real * ca + vv * ymk.imag * sa,
                "Qdp": -V[k] ** 2 * (ykm.imag + bsh) + vv * ykm.imag * ca - vv * ykm.real * sa,
                "Qpd": -V[m] ** 2 * (ymk.imag + bsh) + vv * ymk.imag * ca + vv * ymk.real * sa}


@functools.lru_cache(maxsize=4)
def net_of(name):
    return Net(name)


def _state64(name, cols, case):
    """V, theta, P, Q [S, n] in 64 bits for the packed scenario arrays of one grid."""
    net = net_of(name)
    Pl, Ql, Pg = (c.reshape(-1, net.n) for c in cols)
    b = net.base
    P, Q = Pg - Pl, b["Qg"] - Ql
    if case["limits"]:
        # a single solve takes new injections only: its limit rules read the file's reactive loads
        load = np.broadcast_to(b["Qload"], Ql.shape) if case["kind"] == "solve" else Ql
        V, th = net.newton(P, Q, load, _tol(case))
    else:
        V, th = net.chord(P, Q)
    s = net.injections(V, th)
    return V, th, s.real, s.imag


def exact(case, seed):
    if case["kind"] == "train" or case["grid"] == "c3_base":
        # training: the order of its mini-batches is the library's own; 15,104 buses: a dense 64-bit solve of order
        # 30,000 takes too long
        return None
    gi, cols = inputs(case, seed)
    names = _names(case)
    nbs = np.array([grid_of(n).nB for n in names])
    off = np.concatenate([[0], np.cumsum(nbs[gi])])
    out = {k: np.zeros(off[-1]) for k in ("V", "theta", "Pcalc", "Qcalc")}
    for t, name in enumerate(names):
        mine = np.where(gi == t)[0]
        if not len(mine):
            continue
        at = (off[mine][:, None] + np.arange(nbs[t])[None]).ravel()
        st = _state64(name, [c[at] for c in cols], case)
        for key, v in zip(("V", "theta", "Pcalc", "Qcalc"), st):
            out[key][at] = v.reshape(-1).cpu().numpy()
    if case["kind"] == "solve":
        out.update(net_of(names[0]).flows(st[0][0], st[1][0]))
    return out


# ----------------------------------------------------------------------------------------- the warm start's network
@functools.lru_cache(maxsize=4)
def _linear(name):
    """The grid's base solution and d[V; theta] / d[P; Q] there (float64, host)."""
    net = net_of(name)
    b = net.base
    V, th = net.chord((b["Pg"] - b["Pload"])[None], (b["Qg"] - b["Qload"])[None])
    at = np.concatenate([net.ns, net.n + net.pq])
    J = net.jacobian(V[0], th[0])[torch.as_tensor(at, device=net.dev)][:, torch.as_tensor(at, device=net.dev)]
    return V[0].cpu().numpy(), th[0].cpu().numpy(), at, J, torch.linalg.inv(J)


@functools.lru_cache(maxsize=4)
def _network(name):
    """Weights of a 3 x 512 network with linear skip whose skip is the linearised power flow at the base solution,
    and its normalisation: what a program that serves a trained network loads."""
    V, th, at, _, Ji = _linear(name)
    n = len(V)
    b = grid_of(name).buses()
    sl = sg = SPREAD
    std = np.concatenate([np.hypot(sl * b["Pload"], sg / 3 ** 0.5 * b["Pg"]), sl * np.abs(b["Qload"])])
    scale_in = np.where(std > 0, 1 / np.maximum(std, 1e-30), 0.0)
    scale_out = np.concatenate([np.full(n, 0.005), np.full(n, 0.05)])
    # unknowns [theta; V] at `at` -> outputs [V | theta]; equations [P; Q] at `at` -> features [P | Q]
    rows = np.where(at < n, at + n, at - n)
    S = np.zeros((2 * n, 2 * n))
    S[np.ix_(rows, at)] = Ji.cpu().numpy()
    S = S * std[None, :] / scale_out[:, None]
    rng = np.random.default_rng(7)
    dims = [2 * n, 512, 512, 512, 2 * n]
    params = [(rng.normal(0, (1e-3 if i == 3 else 1.0) / math.sqrt(dims[i]), (dims[i + 1], dims[i])).astype(np.float32),
               np.zeros(dims[i + 1], np.float32)) for i in range(4)]
    params.append((S.astype(np.float32), None))
    mean_in = np.concatenate([b["Pg"] - b["Pload"], b["Qg"] - b["Qload"]])
    return params, [a.astype(np.float32) for a in (mean_in, scale_in, np.concatenate([V, th]), scale_out)]


@functools.lru_cache(maxsize=2)
def _metric(name):
    """A of MLP.set_loss_metric: the linearised mismatch of a predicted start."""
    V, _, at, J, _ = _linear(name)
    n = len(V)
    scale = np.concatenate([np.full(n, 0.005), np.full(n, 0.05)])
    rows = np.where(at < n, at + n, at - n)
    A = np.zeros((2 * n, len(at)))
    A[rows] = scale[rows][:, None] * J.cpu().numpy().T
    return (A * math.sqrt(2 * n / np.sum(A * A))).astype(np.float32)


# -------------------------------------------------------------------------------------------------- prepare, run
def prepare(case, seed):
    st = {"kind": case["kind"]}
    if case["kind"] == "train":
        st["mlp"], st["case"] = _training(case, seed), case
        return st
    gi, cols = inputs(case, seed)
    names = _names(case)
    if case["kind"] == "solve":
        b = grid_of(names[0]).buses()
        st["solver"] = gb.Solver(grid_of(names[0]), **_options(case))
        st["start"] = dict(Pliq=cols[2] - cols[0], Qliq=b["Qg"] - cols[1])
        return st
    st["batch"] = gb.Batch([grid_of(n) for n in names], **_options(case))
    st["inst"], st["cols"] = gi, dict(Pload=cols[0], Qload=cols[1], Pg=cols[2])
    st["out"] = None
    if case["kind"] == "warm":
        params, norm = _network(names[0])
        m = gb.MLP(2 * grid_of(names[0]).nB, 2 * grid_of(names[0]).nB, width=512, n_layers=3, skip=True, seed=1)
        m.set_params(params)
        m.set_norm(*norm)
        st["mlp"] = m
    return st


def _training(case, seed):
    name = case["grid"]
    V, th, at, _, Ji = _linear(name)
    n = len(V)
    dev = _device()
    g = torch.Generator(device=dev).manual_seed(seed)
    b = {k: torch.as_tensor(v, device=dev) for k, v in grid_of(name).buses().items()}
    sl = sg = SPREAD
    shape = (case["rows"], n)
    lf = torch.exp(sl * torch.randn(shape, generator=g, device=dev))
    gf = 1 + sg * (2 * torch.rand(shape, generator=g, device=dev) - 1)
    X = torch.cat([b["Pg"] * gf - b["Pload"] * lf, b["Qg"] - b["Qload"] * lf], 1).double()
    base = torch.cat([b["Pg"] - b["Pload"], b["Qg"] - b["Qload"]])
    rows = torch.as_tensor(np.where(at < n, at + n, at - n), device=dev)
    Y = torch.as_tensor(np.concatenate([V, th]), device=dev).repeat(case["rows"], 1)
    d = ((X - base)[:, torch.as_tensor(at, device=dev)].float() @ Ji.T.float()).double()
    Y[:, rows] += d + 0.3 * d * d
    m = gb.MLP(2 * n, 2 * n, width=case["width"], n_layers=case["layers"], skip=True, seed=seed & 0xffff)
    m.set_data(X.float().cpu().numpy(), Y.float().cpu().numpy())
    if case["metric"]:
        m.set_loss_metric(_metric(name), 1.0)
    return m


def run(st):
    if st["kind"] == "solve":
        s = st["solver"]
        s.set_start(**st["start"])
        r = s.solve()
        return {k: r[k] for k in ("V", "theta", "Pcalc", "Qcalc", "Pdp", "Ppd", "Qdp", "Qpd", "converged",
                                  "iterations", "n_events", "nPQlim", "status")}
    if st["kind"] == "train":
        c, m = st["case"], st["mlp"]
        loss, _ = m.train(c["epochs"], batch=c["batch"], lr=2e-3, lr_final=1e-4, seed=3)
        return {"loss": loss, "params": [a for p in m.params() for a in p if a is not None]}
    b = st["batch"]
    b.set_instances(st["inst"], **st["cols"])
    out = {}
    if st["kind"] == "warm":
        w = b.solve_warm(st["mlp"])
        out = {k: w[k] for k in ("start_kind", "warm_iterations")}
    else:
        b.solve()
    st["out"] = r = b.results(out=st["out"])
    out.update({k: r[k] for k in ("V", "theta", "Pcalc", "Qcalc", "iterations", "status", "n_events")})
    return out


# ----------------------------------------------------------------------------------------------------------- work
@functools.lru_cache(maxsize=None)
def _newton_flops(name, iterations=4):
    """One solve: phasors, injections, Jacobian entries, the block LU and both substitutions."""
    g = grid_of(name)
    a = g.analyse()
    lu = 2 * 24 * a["update_pairs"] + 2 * 12 * a["factor_blocks"] + 30 * a["blocks"]
    return iterations * (40 * g.nB + 8 * g.nnzY + 30 * g.nnzY + lu + 2 * 8 * a["factor_blocks"])


def work(case):
    if case["kind"] == "train":
        n, w, k = 2 * grid_of(case["grid"]).nB, case["width"], case["layers"]
        weights = n * w + (k - 1) * w * w + w * n + n * n
        steps = case["epochs"] * (case["rows"] // case["batch"])
        # forward and weight gradients of every layer, input gradients of all but the first and the skip
        per_row = 2 * (2 * weights + (k - 1) * w * w + w * n)
        if case["metric"]:
            per_row += 4 * n * len(_linear(case["grid"])[2])
        # Adam: gradient-free lower bound of a step, master weights and moments read and written
        return {"bytes": steps * 24 * weights + 4 * weights, "flops": steps * case["batch"] * per_row}
    names = _names(case)
    n = case.get("n", 1)
    nb = sum(grid_of(x).nB for x in names) / len(names) * n
    flops = sum(_newton_flops(x) for x in names) / len(names) * n
    if case.get("dense"):
        flops = 4 * 2 / 3 * (2 * (grid_of(names[0]).nB - 1)) ** 3
    if case["kind"] == "solve":
        return {"bytes": 8 * (2 * nb + 4 * nb + 4 * grid_of(names[0]).nL), "flops": flops}
    if case["kind"] == "warm":
        d = 2 * nb / n
        flops += 2 * n * (2 * d * 512 + 2 * 512 * 512 + d * d)
    return {"bytes": 8 * (3 * nb + 4 * nb) + 16 * n, "flops": flops}
