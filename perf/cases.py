"""The work a user of this engine has it do, as cases that can be timed.

`listed()` names the cases and `draw(rng)` gives more of the same ranges.
`prepare(case, seed)` makes what a program holds before the call (LPs, handles,
networks, host arrays), `run(state)` is one pass through the public entry
points, `work(case)` the arithmetic and traffic that pass cannot do without,
and `exact(case, seed)` the pass's results in 64 bits from plain torch.

The solves end at an iteration cap (or at the tolerance where they reach it
first), so a pass is a fixed amount of work: what a program with a budget of
iterations or a deadline asks for, and the same iterations, check by check,
that a solve to the tolerance is made of.
"""
import math

import numpy as np
import torch

from nirnaya_b200 import batch as B
from nirnaya_b200 import learned
from nirnaya_b200 import lp as L
from nirnaya_b200 import mlp
from nirnaya_b200 import pdhg as P

KINDS = {"random_eq": L.RANDOM_EQ, "zipf": L.ZIPF, "multiperiod": L.MULTIPERIOD, "blend": L.BLEND_FAMILY}
PRECISIONS = {"mixed": P.PREC_MIXED, "fp64": P.PREC_FP64}
WARM_ITERS = 512  # iterations of the earlier solve a family member starts from


def listed():
    return [
        # a small planning LP through the one-call API: the handle is made,
        # used once and freed, so set-up latency is most of it
        dict(name="oneshot_small", path="oneshot", kind="random_eq", m=120, n=300, nnz=2400, iters=1024,
             precision="mixed"),
        # the 2,000 x 5,000 workload, resident: launch latency per iteration
        dict(name="resident_random_eq", path="resident", kind="random_eq", m=2000, n=5000, nnz=40000, iters=2048,
             precision="mixed"),
        # a medium block-angular model in FP64 throughout, odd row count
        dict(name="resident_multiperiod_fp64", path="resident", kind="multiperiod", m=8003, n=20007, nnz=201500,
             iters=1024, precision="fp64"),
        # the 5M-nonzero power-law LP, resident: throughput per iteration
        dict(name="resident_zipf_large", path="resident", kind="zipf", m=200000, n=500000, nnz=5000000, iters=640,
             precision="mixed"),
        # a power-law LP of ordinary size, once, from host arrays
        dict(name="oneshot_zipf", path="oneshot", kind="zipf", m=20000, n=50000, nnz=500000, iters=1024,
             precision="mixed"),
        # a member of the fixed-matrix family: new costs and demands on the
        # resident matrix, started from another member's solution
        dict(name="family_warm", path="family", kind="blend", m=20000, n=50000, nnz=400000, iters=1024,
             precision="mixed"),
        # many block-angular models of uneven sizes in one batch
        dict(name="batch_multiperiod", path="batch", kind="multiperiod", m=500, m_top=20000, count=128, iters=256,
             precision="mixed"),
        # many small LPs in one batch, FP64 throughout
        dict(name="batch_small_fp64", path="batch", kind="random_eq", m=50, m_top=400, count=96, iters=1024,
             precision="fp64"),
        # the reference's own loop, bit for bit
        dict(name="reference_loop", path="reference", kind="random_eq", m=2000, n=5000, nnz=40000, iters=2000,
             precision="fp64"),
        # the solution check of a solved model on the device
        dict(name="verify", path="verify", kind="multiperiod", m=8003, n=20007, nnz=201500, iters=0,
             precision="fp64"),
        # one column network over a family member's variables (ragged count)
        dict(name="predict", path="predict", rows=50001, d_in=16, width=512, depth=3, d_out=8),
        # the warm-start network trained for one epoch from a checkpoint
        dict(name="train", path="train", rows=65536, batch=1024, d_in=16, width=512, depth=3, d_out=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["oneshot", "resident", "resident", "resident", "family", "batch", "batch", "reference",
                       "verify", "predict", "train"])
    if path in ("predict", "train"):
        width = rng.choice([64, 128, 256, 512])
        c = dict(path=path, d_in=rng.choice([16, 24, 64]), width=width, depth=rng.randint(2, 4),
                 d_out=rng.choice([8, 16]))
        if path == "predict":
            return dict(c, rows=_log_int(rng, 64, 60000))
        batch = rng.choice([128, 256, 1024, 2048, 4096])
        return dict(c, rows=batch * rng.randint(4, 16) + rng.randint(0, 99), batch=batch)
    kind = {"family": "blend", "verify": "multiperiod"}.get(path) or rng.choice(["random_eq", "multiperiod", "zipf"])
    precision = "fp64" if path in ("reference", "verify") else rng.choice(["mixed", "mixed", "fp64"])
    if path == "batch":
        kind = rng.choice(["random_eq", "multiperiod"])
        lo = _log_int(rng, 120 if kind == "multiperiod" else 40, 2000)
        return dict(path=path, kind=kind, m=lo, m_top=lo * rng.randint(2, 6), count=rng.randint(5, 64),
                    iters=64 * rng.randint(2, 6), precision=precision)
    m = {"oneshot": (40, 30000), "resident": (40, 120000), "family": (500, 25000), "reference": (40, 10000),
         "verify": (200, 20000)}[path]
    m = _log_int(rng, *m)
    if kind == "multiperiod":
        m = max(m, 120)  # its twelve periods need rows
    # a family's device features and the random families' shapes: n ~ 2.5 m
    n = 5 * (m // 2) + rng.randint(0, 7)
    nnz = {"random_eq": 8 * n, "multiperiod": 10 * n, "zipf": 10 * n, "blend": 8 * n}[kind]
    iters = 0 if path == "verify" else min(_log_int(rng, 200, 3000), max(128, int(2e9 / nnz)))
    return dict(path=path, kind=kind, m=m, n=n, nnz=nnz, iters=iters, precision=precision)


# ------------------------------------------------------------------ inputs

def _lp(case, seed, m=None):
    kind = case["kind"]
    if m is not None:  # a batch member: n follows m
        kw = dict(m=m) if kind == "multiperiod" else dict(m=m, n=5 * m // 2)
    elif kind == "multiperiod":
        kw = dict(m=case["m"], n=case["n"])
    elif kind == "random_eq":
        kw = dict(m=case["m"], n=case["n"])
    else:
        kw = dict(m=case["m"], n=case["n"], target_nnz=case["nnz"])
    return L.generate(KINDS[kind], seed, **kw)


def _batch_lps(case, seed):
    # the members' sizes are the case's, their entries the seed's
    rng = np.random.default_rng([case["m"], case["m_top"], case["count"]])
    ms = np.exp(rng.uniform(math.log(case["m"]), math.log(case["m_top"]), case["count"])).astype(int)
    return [_lp(case, 1000003 * seed + i, m=int(m)) for i, m in enumerate(ms)]


def _family(case, seed):
    """The family, the vectors of the member to solve, and of the earlier one."""
    fam = learned.BlendFamily(case["m"], case["n"], case["nnz"], family_seed=seed)
    now = fam.vectors(*fam.factors(seed + 1))
    before = fam.vectors(*fam.factors(seed + 2))
    return fam, now, before


def _params(case, **kw):
    return P.default_params(max_iters=case["iters"], precision=PRECISIONS[case["precision"]], **kw)


def _net_inputs(case, seed):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((case["rows"], case["d_in"])).astype(np.float32)
    T = np.clip(0.5 + 0.4 * rng.standard_normal((case["rows"], case["d_out"])), 0.0, 1.0).astype(np.float32)
    return X, T


def _dims(case):
    return [case["d_in"]] + [case["width"]] * case["depth"] + [case["d_out"]]


def _weights(case, seed):
    """A network's weights (He-uniform, layer by layer W then b), the layout of Mlp.set_params."""
    rng = np.random.default_rng(seed + 7)
    parts = []
    for a, b in zip(_dims(case), _dims(case)[1:]):
        parts += [rng.uniform(-1.0, 1.0, a * b) * math.sqrt(6.0 / a), 0.1 * rng.standard_normal(b)]
    return np.concatenate(parts).astype(np.float32)


def _net(case, seed):
    net = mlp.Mlp(case["d_in"], case["d_out"], width=case["width"], depth=case["depth"])
    net.set_params(_weights(case, seed))
    return net


def prepare(case, seed):
    path = case["path"]
    s = {"case": case}
    if path == "oneshot":
        s["lp"] = _lp(case, seed)
        s["options"] = P.Options(pdhg_max_iters=case["iters"], pdhg_precision=PRECISIONS[case["precision"]])
    elif path == "resident":
        s["engine"] = P.Engine(_lp(case, seed))
        s["params"] = _params(case)
    elif path == "family":
        fam, (rowlo, cost), (rowlo_b, cost_b) = _family(case, seed)
        s["engine"] = P.Engine(fam.base)
        s["engine"].update_vectors(cost=cost_b, rowlo=rowlo_b)
        x, y, info = s["engine"].solve(P.default_params(max_iters=WARM_ITERS, precision=P.PREC_FP64))
        s.update(cost=cost, rowlo=rowlo, x=x, y=y, omega=info.primal_weight, params=_params(case))
    elif path == "batch":
        s["engine"] = B.BatchEngine(_batch_lps(case, seed))
        s["params"] = _params(case)
    elif path == "reference":
        s["engine"] = P.Engine(_lp(case, seed))
        s["params"] = _params(case, algorithm=P.ALGO_REFERENCE, tol=0.0)
    elif path == "verify":
        lp = _lp(case, seed)
        s["engine"] = P.Engine(lp)
        s["x"] = _near_point(lp, seed)
        s["claimed"] = float(lp.cost @ s["x"])
    elif path == "predict":
        s["net"] = _net(case, seed)
        s["x"] = _net_inputs(case, seed)[0]
    else:
        s["net"] = _net(case, seed)
        s["start"] = _weights(case, seed)  # the checkpoint
        s["net"].set_data(*_net_inputs(case, seed))
    return s


def _near_point(lp, seed):
    """A nearly feasible point, as a solver returns one."""
    return lp.x0 * (1.0 + 1e-7 * np.random.default_rng(seed).standard_normal(lp.ncol))


# -------------------------------------------------------------------- pass

def _solution(x, y, objective, iterations, status):
    return {"x": x, "y": y, "objective": float(objective), "iterations": int(iterations), "status": int(status)}


def run(s):
    case = s["case"]
    path = case["path"]
    if path == "oneshot":
        r = P.PdhgSolver.solve(s["lp"], s["options"])
        return _solution(r.x, r.y, r.objective, r.iterations, r.status)
    if path in ("resident", "reference"):
        x, y, info = s["engine"].solve(s["params"])
        return _solution(x, y, info.objective, info.iterations, info.status)
    if path == "family":
        s["engine"].update_vectors(cost=s["cost"], rowlo=s["rowlo"])
        x, y, info = s["engine"].solve(s["params"], x_init=s["x"], y_init=s["y"], omega_init=s["omega"])
        return _solution(x, y, info.objective, info.iterations, info.status)
    if path == "batch":
        res, _ = s["engine"].solve(s["params"])
        return _solutions([(x, y, i.objective, i.iterations, i.status) for x, y, i in res])
    if path == "verify":
        rep = s["engine"].verify(s["x"], s["claimed"])
        return {k: rep[k] for k in ("passed", "max_bound_viol", "max_row_viol", "max_int_viol", "computed_obj",
                                    "obj_rel_err")}
    if path == "predict":
        return s["net"].predict(s["x"])
    s["net"].set_params(s["start"])
    losses = s["net"].train(1, case["batch"])
    return {"losses": losses, "params": s["net"].get_params()}


def _solutions(results):
    """The members' results of a batch, one array for each quantity."""
    x, y, obj, it, st = zip(*results)
    return {"x": np.concatenate(x), "y": np.concatenate(y), "objective": np.array(obj),
            "iterations": np.array(it, np.int64), "status": np.array(st, np.int64)}


# -------------------------------------------------------------------- work

def work(case):
    path = case["path"]
    if path in ("predict", "train"):
        dims = _dims(case)
        weights = sum(a * b for a, b in zip(dims, dims[1:]))
        rows = case["rows"] if path == "predict" else case["rows"] // case["batch"] * case["batch"]
        if path == "predict":
            return {"bytes": 4.0 * rows * (dims[0] + dims[-1]) + 4.0 * weights, "flops": 2.0 * rows * weights}
        return {"bytes": 4.0 * rows * (dims[0] + dims[-1]) + 8.0 * weights,
                "flops": 2.0 * rows * (3 * weights - dims[0] * dims[1])}
    if path == "batch":
        lo, hi = case["m"], case["m_top"]
        m = case["count"] * (hi - lo) / math.log(hi / lo)  # the mean of the sizes' distribution
        n, nnz = 2.5 * m, 2.5 * m * (10 if case["kind"] == "multiperiod" else 8)
    else:
        m, n, nnz = case["m"], case["n"], case["nnz"]
    # the matrix and the vectors in once, the point out once
    data = 12.0 * nnz + 8.0 * (3 * n + 2 * m) + 8.0 * (n + m)
    # a product and a sum per nonzero and half-iteration, the steps per entry
    return {"bytes": data, "flops": max(1, case["iters"]) * (4.0 * nnz + 12.0 * (n + m))}


# ------------------------------------------------------------------- exact

class _Exact:
    """The PDLP iteration and the reference's loop on one LP, in FP64 torch."""

    def __init__(self, lp, cost=None, rowlo=None):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.from_numpy(np.asarray(a)).to(dev)  # noqa: E731
        m, n = lp.nrow, lp.ncol
        cols = np.repeat(np.arange(n), np.diff(lp.col_start))
        order = np.argsort(lp.row_index, kind="stable")
        row_start = np.concatenate([[0], np.cumsum(np.bincount(lp.row_index, minlength=m))])
        self.rows, self.cols, self.val = t(lp.row_index[order].astype(np.int64)), t(cols[order]), t(lp.value[order])
        self.At_rows, self.At_val = t(lp.row_index.astype(np.int64)), t(lp.value)
        self.At_cols = t(cols)
        self.rp, self.cp = t(row_start), t(lp.col_start)
        self.m, self.n, self.offset = m, n, lp.obj_offset
        bound = lambda v, fill: torch.where(torch.isfinite(v) & (v.abs() < 1e20), v, torch.full_like(v, fill))  # noqa: E731
        self.c = t(lp.cost if cost is None else cost)
        self.l, self.u = bound(t(lp.collo), -math.inf), bound(t(lp.colup), math.inf)
        self.rl = bound(t(lp.rowlo if rowlo is None else rowlo), -math.inf)
        self.ru = bound(t(lp.rowup), math.inf)
        fin = lambda v: torch.where(torch.isfinite(v), v.abs(), torch.zeros_like(v))  # noqa: E731
        self.b = torch.maximum(fin(self.rl), fin(self.ru))

    def matrices(self, dr, dc):
        a = torch.sparse_csr_tensor(self.rp, self.cols, self.val * dr[self.rows] * dc[self.cols], (self.m, self.n))
        at = torch.sparse_csr_tensor(self.cp, self.At_rows, self.At_val * dr[self.At_rows] * dc[self.At_cols],
                                     (self.n, self.m))
        return a, at

    def scales(self):
        """Ten Ruiz passes and a Pock-Chambolle pass, rounded to powers of two."""
        dr, dc = torch.ones_like(self.rl), torch.ones_like(self.c)
        for k in range(11):
            w = self.val.abs() * dr[self.rows] * dc[self.cols]
            how = "amax" if k < 10 else "sum"
            sr = torch.zeros_like(dr).scatter_reduce_(0, self.rows, w, how)
            sc = torch.zeros_like(dc).scatter_reduce_(0, self.cols, w, how)
            dr = torch.where(sr > 0, dr / sr.sqrt(), dr)
            dc = torch.where(sc > 0, dc / sc.sqrt(), dc)

        def pow2(d):
            f, e = torch.frexp(d)
            e = torch.where(f >= math.sqrt(0.5), e, e - 1).clamp(-60, 60)
            return torch.ldexp(torch.ones_like(d), e)

        return pow2(dr), pow2(dc)

    def norm(self, a, at):
        """||A||_2 by 64 rounds of power iteration from a hashed start."""
        with np.errstate(over="ignore"):
            z = np.arange(self.n, dtype=np.uint64) * np.uint64(0x9e3779b97f4a7c15) + np.uint64(0x632be59bd9b4e019)
            z = (z ^ (z >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
            z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
            z ^= z >> np.uint64(31)
        u = torch.from_numpy(0.5 + (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53).to(self.c.device)
        u = u / u.norm()
        for _ in range(64):
            w = at @ (a @ u)
            nrm = w.norm()
            u = w / nrm
        return math.sqrt(float(nrm))

    def pdlp(self, iters, tol=1e-6, x=None, y=None, omega=None, K=64):
        dr, dc = self.scales()
        a, at = self.matrices(dr, dc)
        c, l, u, rl, ru = self.c * dc, self.l / dc, self.u / dc, self.rl * dr, self.ru * dr
        eta = 0.998 / max(self.norm(a, at), 1e-30)
        cn, bn = float(c.norm()), float((self.b * dr).norm())
        omega0 = cn / bn if cn > 1e-10 and bn > 1e-10 else 1.0
        omega0 = omega = omega or omega0
        x = torch.zeros_like(c) if x is None else torch.from_numpy(x).to(c.device) / dc
        x = torch.minimum(torch.maximum(x, l), u)
        y = torch.zeros_like(rl) if y is None else torch.from_numpy(y).to(c.device) / dr
        x0, y0 = x, y
        bnorm, cnorm = float(self.b.norm()), float(self.c.norm())
        it, k_base, r_anchor, r_prev, status = 0, 0, None, 0.0, 6
        zero = torch.zeros((), dtype=torch.float64, device=c.device)
        while it < iters:
            tau, sigma = eta / omega, eta * omega
            for i in range(K):
                k = k_base + i
                w, v = (k + 1.0) / (k + 2.0), 1.0 / (k + 2.0)
                xk, yk = x, y
                xp = torch.minimum(torch.maximum(xk - tau * (c - at @ yk), l), u)
                ax = a @ (2.0 * xp - xk)
                yp = yk + sigma * (torch.minimum(torch.maximum(ax - yk / sigma, rl), ru) - ax)
                x = w * (2.0 * xp - xk) + v * x0
                y = w * (2.0 * yp - yk) + v * y0
            it += K
            # relative KKT error of (xp, yp) in the LP's own space
            ax, rc = (a @ xp) / dr, self.c - (at @ yp) / dc
            xo, yo = xp * dc, yp * dr
            lam = torch.where(((rc > 0) & torch.isfinite(self.l)) | ((rc < 0) & torch.isfinite(self.u)), rc, zero)
            wrong = torch.where(((yo > 0) & ~torch.isfinite(self.rl)) | ((yo < 0) & ~torch.isfinite(self.ru)), yo, zero)
            pres = ax - torch.minimum(torch.maximum(ax, self.rl), self.ru)
            xv = xo - torch.minimum(torch.maximum(xo, self.l), self.u)
            d_row = torch.where(yo > 0, self.rl, self.ru) * yo
            d_col = torch.where(lam > 0, self.l, self.u) * lam
            dobj = float(torch.where((yo != 0) & (wrong == 0), d_row, zero).sum()
                         + torch.where(lam != 0, d_col, zero).sum()) + self.offset
            pobj = float(self.c @ xo) + self.offset
            kkt = max(math.sqrt(float(pres @ pres + xv @ xv)) / (1 + bnorm),
                      math.sqrt(float((rc - lam) @ (rc - lam) + wrong @ wrong)) / (1 + cnorm),
                      abs(pobj - dobj) / (1 + abs(pobj) + abs(dobj)))
            if kkt <= tol:
                status = 0
                break
            dx, dy = float((xk - xp).norm()), float((yk - yp).norm())
            res = math.sqrt(omega * dx * dx + dy * dy / omega)
            if r_anchor is None:
                r_anchor, restart = res, k_base + K >= 0.36 * it
            else:
                restart = res <= 0.2 * r_anchor or (res <= 0.8 * r_anchor and res > r_prev) or k_base + K >= 0.36 * it
            r_prev = res
            k_base += K
            if restart and it < iters:
                dxa, dya = float((xp - x0).norm()), float((yp - y0).norm())
                if dxa > 1e-10 and dya > 1e-10:
                    lw = 0.5 * math.log(dya / dxa) + 0.5 * math.log(omega)
                    ten = math.log(10.0)
                    lw = min(max(lw, math.log(omega) - ten), math.log(omega) + ten)
                    omega = math.exp(min(max(lw, math.log(omega0) - ten), math.log(omega0) + ten))
                x = x0 = xp
                y = y0 = yp
                k_base, r_anchor = 0, res
        x, y = (xp * dc).cpu().numpy(), (yp * dr).cpu().numpy()
        return _solution(x, y, float(self.c.cpu().numpy() @ x) + self.offset, it, status), omega

    def reference(self, iters):
        one_r, one_c = torch.ones_like(self.rl), torch.ones_like(self.c)
        a, at = self.matrices(one_r, one_c)
        v = one_c
        for _ in range(12):
            w = at @ (a @ v)
            nrm = math.sqrt(max(1e-12, float(w @ w)))
            v = w / nrm
        step = 0.85 / max(1e-6, math.sqrt(nrm))
        lf, uf = torch.isfinite(self.l), torch.isfinite(self.u)
        x = torch.where(lf & uf, 0.5 * (self.l + self.u),
                        torch.where(lf, self.l.clamp(min=0.0), torch.where(uf, self.u.clamp(max=0.0), 0.0 * self.c)))
        y = 0.0 * self.rl
        status, done = 6, iters
        for it in range(iters):
            xn = torch.minimum(torch.maximum(x - step * (self.c - at @ y), self.l), self.u)
            ax = a @ (2.0 * xn - x)
            x = xn
            y = y + step * (torch.minimum(torch.maximum(ax - y / step, self.rl), self.ru) - ax)
            if it > 20 and it % 32 == 0 and float(torch.maximum(self.rl - ax, ax - self.ru).max()) <= 1e-6:
                status, done = 0, it + 1
                break
        x, y = x.cpu().numpy(), y.cpu().numpy()
        return _solution(x, y, float(self.c.cpu().numpy() @ x) + self.offset, done, status)


def exact(case, seed):
    path = case["path"]
    if path in ("oneshot", "resident"):
        return _Exact(_lp(case, seed)).pdlp(case["iters"])[0]
    if path == "family":
        fam, (rowlo, cost), (rowlo_b, cost_b) = _family(case, seed)
        old, omega = _Exact(fam.base, cost_b, rowlo_b).pdlp(WARM_ITERS)
        return _Exact(fam.base, cost, rowlo).pdlp(case["iters"], x=old["x"], y=old["y"], omega=omega)[0]
    if path == "batch":
        rs = [_Exact(lp).pdlp(case["iters"])[0] for lp in _batch_lps(case, seed)]
        return _solutions([(r["x"], r["y"], r["objective"], r["iterations"], r["status"]) for r in rs])
    if path == "reference":
        return _Exact(_lp(case, seed)).reference(case["iters"])
    if path == "verify":
        lp = _lp(case, seed)
        x = _near_point(lp, seed)
        e = _Exact(lp)
        fin = np.isfinite
        # the row activities in extended precision: the violations are small differences of them
        ax = np.zeros(lp.nrow, np.longdouble)
        cols = np.repeat(np.arange(lp.ncol), np.diff(lp.col_start))
        np.add.at(ax, lp.row_index, lp.value.astype(np.longdouble) * x[cols])

        def viol(v, lo, hi):
            lo, hi = lo.cpu().numpy(), hi.cpu().numpy()
            out = np.zeros(1)
            for d, b in ((lo - v, lo), (v - hi, hi)):
                ok = fin(b)
                out = np.append(out, (np.maximum(d[ok], 0) / (1 + np.abs(b[ok]))).astype(np.float64))
            return float(out.max())

        obj = float((lp.cost.astype(np.longdouble) * x).sum() + lp.obj_offset)
        rows, box = viol(ax, e.rl, e.ru), viol(x, e.l, e.u)
        return {"passed": None, "max_bound_viol": box, "max_row_viol": rows, "max_int_viol": 0.0,
                "computed_obj": obj, "obj_rel_err": None}
    if path == "predict":
        p, dims = _weights(case, seed).astype(np.float64), _dims(case)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        h = torch.from_numpy(_net_inputs(case, seed)[0].astype(np.float64)).to(dev)
        o = 0
        for i, (a, b) in enumerate(zip(dims, dims[1:])):
            w = torch.from_numpy(p[o:o + a * b].reshape(b, a)).to(dev)
            bias = torch.from_numpy(p[o + a * b:o + a * b + b]).to(dev)
            o += a * b + b
            h = h @ w.T + bias
            if i < len(dims) - 2:
                h = h.clamp(min=0.0)
        return h.cpu().numpy()
    # a training epoch: the order of the samples is the library's own
    return None
