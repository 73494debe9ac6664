"""The work that users of this package have it do, as timed cases.

A case names one call on a synthetic employer-employee panel: what the call
is (`kind`), the panel (workers, firms, years, the spell's range of years, the
yearly probability of a move, how many covariates, weights or not, with or
without year effects, and `set`: "all" rows, the largest "connected" set, the
"core" of it with at least two partners each, or a "linked" panel, which is
leave-one-out connected as drawn) and the call's own options.  The panels
follow `simulate.py`'s specification and are drawn on the GPU here; the sizes
are those of the package's own presets, tests and benchmark and the range
between them.

`exact` solves the same problems in plain torch, in 64 bits: sparse products
with the group incidence and a conjugate gradient run to rounding.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from hdfe_stream_b200 import adjoint, batch, connected, fit, gpu, inference, pass0
from hdfe_stream_b200.leaveout import TRACE_SEED_OFFSET, InverseOperator
from hdfe_stream_b200.simulate import Rows

F64 = torch.float64
PANEL = dict(years=10, lo=7, hi=10, move=0.1, cov=2, weights=False, year_fe=True, set="all")


def _case(name, kind, workers, firms, **options):
    return {"name": name, "kind": kind, "workers": workers, "firms": firms, **PANEL, **options}


def listed():
    return [
        # the smallest fits: a quick look at a small panel, one of many subsamples;
        # launches and host reads count, not bytes
        _case("fit_20k", "fit", 20_000, 2_000, lo=8, hi=8),
        # an ordinary weighted fit (3.4M rows), not restricted: many components
        _case("fit_400k_weighted", "fit", 400_000, 40_000, weights=True),
        # the benchmark's fit: 5M workers over 15 years, the largest connected
        # set after min_degree 2 (about 20M rows are left)
        _case("fit_5m", "fit", 5_000_000, 500_000, years=15, lo=5, hi=12, move=0.08,
              set="core"),
        # the same path from pinned host rows to host effects, bound by the bus
        _case("fit_host_1m", "fit_host", 1_000_000, 100_000, years=15, lo=5, hi=12, move=0.08),
        # the solver seam as a host program drives it: its S, one block of 8
        # right-hand sides, host arrays in and out, warm-started
        _case("solve_400k_k8", "solve", 400_000, 40_000, k=8, warm=True),
        # beta and its iid, HC1 and clustered variances after a fit
        _case("estimate_400k_weighted", "estimate", 400_000, 40_000, weights=True),
        # gradients through a fit: forward, and backward for two objectives
        _case("adjoint_400k_weighted", "adjoint", 400_000, 40_000, weights=True, set="linked"),
        # every row's leverage, the default number of draws (250: a ragged last block)
        _case("leverages_100k", "leverages", 100_000, 10_000, year_fe=False, set="linked",
              draws=250, block=32),
        # the KSS leave-out variance components of the benchmark (8M rows)
        _case("kss_1m", "kss", 1_000_000, 100_000, year_fe=False, set="linked",
              draws=256, block=32),
        # many small regressions of uneven size in one launch
        _case("batch_24", "batch", 20_000, 2_000, lo=8, hi=8, systems=24, set="linked"),
        # raw id columns in any order to coded, sorted rows (8.5M)
        _case("pass0_1m", "pass0", 1_000_000, 100_000),
        # the leave-one-out connected set of a 1M-worker network
        _case("connected_1m", "connected", 1_000_000, 100_000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "fit_host", "solve", "estimate", "adjoint",
                       "leverages", "kss", "batch", "pass0", "connected"])
    most = {"fit": 4_000_000, "fit_host": 2_000_000, "solve": 1_000_000, "estimate": 2_000_000,
            "adjoint": 1_000_000, "leverages": 400_000, "kss": 400_000, "batch": 60_000,
            "pass0": 2_000_000, "connected": 2_000_000}[kind]
    least = 5_000 if kind in ("batch", "fit", "leverages", "kss") else 20_000
    workers = _log(rng, least, most)
    years = rng.choice([6, 10, 13, 15, 22])
    lo = rng.randint(3, years - 1)
    case = {"kind": kind, "workers": workers, "firms": max(workers // rng.randint(8, 16), 100),
            **PANEL, "years": years, "lo": lo, "hi": rng.randint(lo, min(years, 12, lo + 5))
            if lo <= 12 else lo, "move": round(rng.uniform(0.08, 0.2), 3),
            "cov": rng.choice([1, 2, 2, 3]), "weights": rng.random() < 0.4}
    if kind in ("fit", "estimate"):
        case.update(year_fe=rng.random() < 0.8,
                    set=rng.choice(["all", "connected", "core", "linked"]))
    if kind == "solve":
        case.update(k=rng.randint(1, 20), warm=rng.random() < 0.5)
    if kind == "adjoint":
        case.update(set="linked")
    if kind in ("leverages", "kss"):
        case.update(set="linked", year_fe=False, draws=rng.randint(40, 250),
                    block=rng.choice([8, 16, 32, 32]))
    if kind == "kss":
        case.update(weights=False)
    if kind == "batch":
        case.update(set="linked", systems=rng.randint(4, 40))
    return case


# ------------------------------------------------------------------ panels


def _panel(case, seed):
    """One panel in pass 0's layout as plain torch tensors: g (N,), codes
    (N, D) int64, V (m, N), w (N,) or None, n_levels, and the groups' count."""
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)

    def normal(n, sd=1.0):
        return sd * torch.randn(n, generator=gen, device=dev, dtype=F64)

    def uniform(n):
        return torch.rand(n, generator=gen, device=dev, dtype=F64)
    n, nf, ny = case["workers"], case["firms"], case["years"]
    length = case["lo"] + torch.randperm(n, generator=gen, device=dev) % (
        case["hi"] - case["lo"] + 1)
    alpha, psi, tau = normal(n), normal(nf, 0.5), normal(ny, 0.1)
    first = (uniform(n) * (ny - length + 1)).long()
    age0 = 25 + (uniform(n) * (36 - length)).long()
    worker = torch.repeat_interleave(torch.arange(n, device=dev), length)
    N = worker.numel()
    i = torch.arange(N, device=dev)
    t = i - (torch.cumsum(length, 0) - length)[worker]
    year, age = first[worker] + t, (age0[worker] + t).to(F64)
    a = alpha[worker]
    score = 0.3 * a + math.sqrt(1 - 0.09) * normal(N)
    rank = (torch.special.ndtr(score) * nf).long().clamp(max=nf - 1)
    starts = (t == 0) | (uniform(N) < case["move"])
    pick = torch.argsort(psi)[rank]
    if case["set"] == "linked":
        # one worker in so many is hired away in mid-spell, four into every firm,
        # which makes the network leave-one-out connected at a fixed size
        at = (torch.cumsum(length, 0) - length // 2)[:4 * nf]
        pick[at], starts[at] = torch.arange(4 * nf, device=dev) % nf, True
        starts[at + 1] = (t == 0)[at + 1]
    last = torch.cummax(torch.where(starts, i, torch.zeros_like(i)), 0).values
    firm = pick[last]
    X = [age * age / 100, age * age * age / 1000]
    X += [normal(N) + 0.5 * a for _ in range(2, case["cov"])]
    y = 10 + a + psi[firm] + tau[year] + 0.08 * X[0] - 0.012 * X[1] + normal(N, 0.5)
    V = torch.stack([y] + X[:case["cov"]])
    w = 0.5 + 1.5 * uniform(N) if case["weights"] else None
    order = torch.argsort((worker * nf + firm) * ny + year)
    worker, firm, year, V = worker[order], firm[order], year[order], V[:, order]
    w = None if w is None else w[order]
    if case["set"] in ("core", "connected"):    # as a user's pass 0 restricts the rows
        f, g, k = firm.to(torch.int32), worker.to(torch.int32), 1 + (case["set"] == "core")
        alive = connected.pair_components(g, f, n, nf, (k, k))[0] == 0
        keep = alive[worker] & alive[n + firm]
        worker, firm, year, V = worker[keep], firm[keep], year[keep], V[:, keep]
        w = None if w is None else w[keep]
    left, g = torch.unique_consecutive(worker, return_inverse=True)
    fes = [firm, year] if case["year_fe"] else [firm]
    return SimpleNamespace(g=g, codes=torch.stack(fes, 1), V=V.contiguous(), w=w,
                           n_levels=[nf, ny][:len(fes)], G=len(left), gen=gen)


def _rows(p):
    return fit.DeviceRows(p.g.to(torch.int32), p.codes.to(torch.int32).contiguous(), p.V, p.w,
                          list(p.n_levels), [f"v{j}" for j in range(p.V.shape[0])])


def _systems(case, seed):
    """The batch's panels: workers log-uniform from a quarter of the case's up."""
    out = []
    for s in range(case["systems"]):
        n = int(case["workers"] * math.exp(math.log(0.25) * (0.618034 * s % 1.0)))
        out.append(_panel({**case, "workers": n, "firms": n // 10}, seed * 1000 + s))
    return out


def _raw(case, seed):
    """Unsorted raw columns: sparse worker, firm and year ids, V (N, m), w."""
    p = _panel({**case, "set": "linked"}, seed)
    mix = torch.randperm(len(p.g), generator=p.gen, device=p.g.device)
    spread = torch.randperm(4 * p.G, generator=p.gen, device=p.g.device)[:p.G]
    worker, codes = spread[p.g][mix].to(torch.int32), p.codes[mix].to(torch.int32)
    fes = [codes[:, 0] * 3 + 1000] + ([codes[:, 1] + 1995] if case["year_fe"] else [])
    return worker, fes, p.V.T[mix].contiguous(), None if p.w is None else p.w[mix]


def _right_sides(case, p):
    """k right-hand sides of the reduced system in S's range, D'W M r, and the
    warm start of a solve whose weights moved a little."""
    R = torch.randn((len(p.g), case["k"]), generator=p.gen, device=p.g.device, dtype=F64)
    m = _Plain(p)
    B = m.levels(m.center(R))
    X0 = torch.randn(B.shape, generator=p.gen, device=p.g.device, dtype=F64) if case["warm"] \
        else None
    return B, X0


# ------------------------------------------------------------------ the calls


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems = [Rows(gcode=p.g.cpu().numpy().astype(np.uint32),
                        codes=p.codes.cpu().numpy().astype(np.uint32),
                        V=np.ascontiguousarray(p.V.T.cpu().numpy()),
                        w=None if p.w is None else p.w.cpu().numpy(), n_levels=p.n_levels,
                        n_groups=p.G, names=[]) for p in _systems(case, seed)]
        b = batch.concat(systems)
        return case, b, fit.DeviceRows.from_rows(b.rows)
    if kind == "pass0":
        return case, _raw(case, seed)
    p = _panel(case, seed)
    rows = _rows(p)
    if kind == "fit":
        return case, rows
    if kind == "fit_host":
        def pin(t):
            return None if t is None else t.cpu().pin_memory()
        return case, pin(rows.gcode), pin(rows.codes), pin(rows.V), pin(rows.w), rows.n_levels
    if kind == "connected":
        return case, rows.gcode, rows.codes[:, 0].contiguous(), p.G, p.n_levels[0]
    if kind == "adjoint":
        return case, rows.V[0].clone(), p.w, rows.gcode, rows.codes, p.V[1:].T, p.n_levels
    if kind == "solve":
        cells = fit.pass1(rows)
        S = fit.build_s(cells)
        S = SimpleNamespace(indptr=S.indptr.cpu().numpy(), indices=S.indices.cpu().numpy(),
                            data=S.data.cpu().numpy())
        solve, _ = gpu.explicit_solver(S, fit.jacobi(cells.diag).cpu().numpy(), 1e-10, 5000)
        B, X0 = _right_sides(case, p)
        return case, solve, B.cpu().numpy(), None if X0 is None else X0.cpu().numpy()
    res = fit.fit(rows)
    if kind == "estimate":
        return case, rows, res
    op = InverseOperator(rows, res.cells, res.S, rows.V[1:].T)
    return case, op, res


def run(state):
    case, rest = state[0], state[1:]
    kind = case["kind"]
    if kind == "fit":
        return fit.fit(rest[0]).gamma
    if kind == "fit_host":
        gcode, codes, V, w, n_levels = rest
        return fit.fit_host(gcode, codes, V, n_levels, w=w).gamma.cpu()
    if kind == "solve":
        solve, B, X0 = rest
        return solve(B, np.zeros(case["k"], bool), X0)[0]
    if kind == "estimate":
        rows, res = rest
        e = inference.estimate(rows, res.cells, res.gamma, clusters=("fe1",))
        return {"beta": e["beta"], "rss": e["rss"], "k_fe": e["k_fe"], **e["vcov"]}
    if kind == "adjoint":
        y, w, gcode, codes, X, n_levels = rest
        y = y.detach().requires_grad_(True)
        w = w.detach().requires_grad_(True) if w is not None else None
        on = (y,) if w is None else (y, w)
        beta, gamma, alpha, _ = adjoint.FixedEffectsSolve.apply(y, w, gcode, codes, X, n_levels)
        comp = adjoint.plug_in_components(gamma, alpha, w, gcode, codes, n_levels)
        g1 = torch.autograd.grad(comp[0], on, retain_graph=True)
        g2 = torch.autograd.grad(beta[0], on)
        return {"beta": beta.detach(), "components": comp.detach(), "var_psi": list(g1),
                "beta0": list(g2)}
    if kind == "leverages":
        lev = rest[0].jla_leverages(case["draws"], case["block"], seed=11)
        return [lev.leverage, lev.complement, lev.factor]
    if kind == "kss":
        op, res = rest
        r = op.leave_out_components(res, case["draws"], case["block"], seed=11)
        return {"leverage": r.leverages.leverage, "complement": r.leverages.complement,
                "factor": r.leverages.factor, "sigma2": r.diagnostics["sigma2"],
                "plug_in": list(r.plug_in.values()), "bias": list(r.bias.values()),
                "leave_out": list(r.leave_out.values())}
    if kind == "batch":
        solver = batch.BatchSolver(rest[0], drows=rest[1])
        X, _ = solver.solve()
        return solver.gammas(solver.normalize(X))
    if kind == "pass0":
        worker, fes, V, w = rest[0]
        rows, levels = pass0.pass0(worker, fes, V, w)
        return [rows.gcode, rows.codes, rows.V, rows.w, levels]
    alive, info = connected.leave_one_out(*rest)
    return [alive, info["rows"], info["rounds"]]


def work(case):
    """Each input read once and each output written once; the additions and
    multiplications of one visit to every row (for each draw, where a call
    has draws)."""
    N = case["workers"] * (case["lo"] + case["hi"]) / 2
    D, m, L = 1 + case["year_fe"], 1 + case["cov"], case["firms"]
    row = 4 + 4 * D + 8 * m + 8 * case["weights"]
    kind, draws, passes, out = case["kind"], 1, 1, 8 * L * m
    if kind == "batch":
        N, L = N * case["systems"] / 2, L * case["systems"] / 2
        out = 8 * L * m
    elif kind == "solve":
        row, out, passes = 4, 24 * L * case["k"], case["k"]
    elif kind == "estimate":
        out = 64 * m * m
    elif kind == "adjoint":
        out, passes = 16 * N * (1 + case["weights"]), 4
    elif kind in ("leverages", "kss"):
        draws = case["draws"] * (3 if kind == "kss" else 1)
        out, passes = 8 * N * (4 if kind == "kss" else 3), 4
    elif kind == "pass0":
        out = row * N
    elif kind == "connected":
        row, out = 8, case["workers"] + L
    return {"bytes": row * N + out, "flops": 2 * N * (D + 1) * m * passes * draws}


# ------------------------------------------------------------------ in 64 bits, plain


class _Plain:
    """The weighted least-squares problem of a panel: sums over groups and
    levels, the reduced matrix S = D'WD - F' diag(1/n) F as sparse products,
    and S^- by a conjugate gradient run to rounding."""

    def __init__(self, p, covariates=False):
        dev = p.g.device
        self.g, self.G, self.p = p.g, p.G, p
        self.w = torch.ones(len(p.g), dtype=F64, device=dev) if p.w is None else p.w
        offs = np.concatenate(([0], np.cumsum(p.n_levels)))
        self.L = int(offs[-1])
        self.offs = [int(o) for o in offs]
        self.lev = [p.codes[:, d] + self.offs[d] for d in range(p.codes.shape[1])]
        self.gw = self._sum(self.g, self.w[:, None], self.G)
        self.obs = sum(self._sum(l, self.w[:, None], self.L) for l in self.lev)[:, 0]
        self.X = p.V[1:].T if covariates else self.w.new_zeros((len(p.g), 0))
        # sums of weights per (group, level), and per pair of levels
        self.F = [self._sparse(self.g, l, (self.G, self.L)) for l in self.lev]
        self.T = [self._sparse(l, self.g, (self.L, self.G)) for l in self.lev]
        self.off = [self._sparse(a, b, (self.L, self.L)) for a in self.lev for b in self.lev
                    if a is not b]
        diag = self.obs.clone()
        for t in self.T:
            diag -= (torch.sparse_csr_tensor(t.crow_indices(), t.col_indices(), t.values() ** 2,
                                             t.shape) @ (1 / self.gw))[:, 0]
        self.dinv = torch.where(diag > 1e-12, 1 / diag, 0.0)
        self._border = None

    @staticmethod
    def _sum(idx, x, n):
        return x.new_zeros((n, x.shape[1])).index_add_(0, idx, x)

    def gather(self, U):
        return sum(U[l] for l in self.lev)

    def levels(self, R):
        R = self.w[:, None] * R
        return sum(self._sum(l, R, self.L) for l in self.lev)

    def groups(self, R):
        return self._sum(self.g, self.w[:, None] * R, self.G)

    def center(self, R):
        return R - (self.groups(R) / self.gw)[self.g]

    def _sparse(self, i, j, shape):
        A = torch.sparse_coo_tensor(torch.stack([i, j]), self.w, shape).coalesce()
        return A.to_sparse_csr()

    def S(self, P):
        u = sum(f @ P for f in self.F) / self.gw
        return self.obs[:, None] * P + sum(o @ P for o in self.off) - sum(t @ u for t in self.T)

    def solve(self, B, X0=None):
        X = torch.zeros_like(B) if X0 is None else X0.clone()
        R = B - self.S(X) if X0 is not None else B.clone()
        d = self.dinv[:, None]
        P = R * d
        rz, norm = (R * P).sum(0), torch.linalg.vector_norm(B, dim=0).clamp(min=1e-300)
        best, since = float("inf"), 0
        live = torch.ones_like(norm, dtype=torch.bool)
        while since < 40 and bool(live.any()):
            Q = self.S(P)
            pq = (P * Q).sum(0)
            a = torch.where(live & (pq > 0), rz / pq, 0.0)
            X += a * P
            R -= a * Q
            rel = torch.linalg.vector_norm(R, dim=0) / norm
            live &= rel > 1e-14
            worst = float(rel.max())
            best, since = (worst, 0) if worst < 0.5 * best else (best, since + 1)
            Z = R * d
            new = (R * Z).sum(0)
            P = Z + torch.where(live, new / rz, 0.0) * P
            rz = new
        return X

    def inverse(self, levels, cov, streamed):
        """u = (A'WA)^- v for v = (levels, cov, streamed): (U, C, U_g)."""
        rhs = levels - self._from_groups(streamed)
        if self._border is None and self.X.shape[1]:
            xc = self.center(self.X)
            T = self.levels(xc)
            Z = self.solve(T)
            self._border = Z, self.X.T @ (self.w[:, None] * xc) - T.T @ Z
        U, C = self.solve(rhs), rhs.new_zeros((0, rhs.shape[1]))
        if self.X.shape[1]:
            Z, schur = self._border
            rhs_x = cov - self.groups(self.X).T @ (streamed / self.gw)
            C = torch.linalg.solve(schur, rhs_x - Z.T @ rhs)
            U = U - Z @ C
        R = self.gather(U) + self.X @ C
        return U, C, (streamed - self.groups(R)) / self.gw

    def _from_groups(self, streamed):
        return self.levels((streamed / self.gw)[self.g])

    def rows(self, U, C, Ug):
        return self.gather(U) + self.X @ C + Ug[self.g]

    def reduce(self, R):
        return self.levels(R), self.X.T @ (self.w[:, None] * R), self.groups(R)

    def project(self, R):
        return self.rows(*self.inverse(*self.reduce(R)))

    def components(self):
        """Per level of the first dimension its component's smallest level."""
        f, n = self.lev[0], self.p.n_levels[0]
        lab = torch.arange(n, device=f.device)
        while True:
            low = torch.full((self.G,), n, device=f.device).scatter_reduce_(
                0, self.g, lab[f], "amin")
            new = lab.scatter_reduce(0, f, low[self.g], "amin")
            new = new[new]
            if bool((new == lab).all()):
                return lab
            lab = new

    def normalize(self, U):
        U, n0 = U.clone(), self.p.n_levels[0]
        root, w = self.components(), self.obs[:, None]
        mean = self._sum(root, w[:n0] * U[:n0], n0) / self._sum(root, w[:n0], n0).clamp(
            min=1e-300)
        U[:n0] -= mean[root]
        for a, b in zip(self.offs[1:-1], self.offs[2:]):
            U[a:b] -= (w[a:b] * U[a:b]).sum(0) / w[a:b].sum()
        return U

    def fixed_effects(self):
        return self.normalize(self.solve(self.levels(self.center(self.p.V.T))))

    def regression(self):
        """beta, the normalised effects net of the covariates, alpha, residuals."""
        gamma = self.fixed_effects()
        V = self.center(self.p.V.T - self.gather(gamma))
        A = V.T @ (self.w[:, None] * V)
        beta = torch.linalg.solve(A[1:, 1:], A[1:, 0])
        gam = gamma[:, 0] - gamma[:, 1:] @ beta
        part = self.p.V[0] - self.p.V[1:].T @ beta - self.gather(gam[:, None])[:, 0]
        alpha = self.groups(part[:, None])[:, 0] / self.gw[:, 0]
        return beta, gam, alpha, part - alpha[self.g], V


def _signs(n, first, count, seed, device):
    """+-1 by a splitmix64 hash of (seed, position, draw)."""
    def wrap(v):
        v &= 2 ** 64 - 1
        return v - 2 ** 64 if v >= 2 ** 63 else v

    def shift(x, k):
        return (x >> k) & (2 ** (64 - k) - 1)
    c1, c2 = wrap(0xBF58476D1CE4E5B9), wrap(0x94D049BB133111EB)
    i = torch.arange(n, device=device)[:, None] * wrap(0x9E3779B97F4A7C15)
    j = torch.arange(first, first + count, device=device)[None, :] * c1
    x = i ^ j ^ wrap(seed)
    x = (x ^ shift(x, 30)) * c1
    x = (x ^ shift(x, 27)) * c2
    x = x ^ shift(x, 31)
    return torch.where(x >= 0, 1.0, -1.0).to(F64)


def _leverages(m, draws, seed):
    N, root = len(m.g), torch.sqrt(m.w)[:, None]
    mom = m.w.new_zeros((5, N))
    for a in range(0, draws, 32):
        r = _signs(N, a, min(32, draws - a), seed, m.g.device)
        proj = root * m.project(r / root)
        P, M = proj ** 2, (r - proj) ** 2
        for slot, v in zip(mom, (P, M, P * P, M * M, P * M)):
            slot += v.sum(1)
    P, M, pp, mm, pm = mom / draws
    lev = P / (P + M)
    com = 1 - lev
    V = (com ** 2 * pp + lev ** 2 * mm - 2 * lev * com * pm) / draws
    B = (com * pp - lev * mm + (com - lev) * pm) / draws
    return lev, com, 1 - V / com ** 2 + B / com


def _trace(m, sigma2, draws, seed):
    """The bias of var(psi), var(alpha) and cov(psi, alpha), one dimension."""
    L, G, c, N = m.L, m.G, m.X.shape[1], len(m.g)
    f, total = m.lev[0], m.w.new_zeros(8)

    def drop(levels, streamed):
        off = (streamed.sum(0) - levels.sum(0)) / (L + G)
        return levels + off, streamed - off
    for at in range(0, draws, 32):
        z = _signs(L + G + c, at, min(32, draws - at), seed, m.g.device)
        zl, zg = z[:L], z[L:L + G]
        dl, dg = drop(zl, zg)
        row = m.rows(*m.inverse(dl, z[L + G:], dg)) * sigma2[:, None]
        vl, vx, vg = m.reduce(row)
        vl, vg = drop(vl, vg)
        U, _, Ug = m.inverse(vl, vx, vg)
        a1, a2, b1, b2 = zl[f], U[f], zg[m.g], Ug[m.g]
        k = a1.shape[1]
        total += torch.stack([m.w.sum() * k, (a1 * a2).sum(), (b1 * b2).sum(),
                              (a1 * b2 + b1 * a2).sum(), *(0 * total[:4])])
        means = [x.sum(0) for x in (a1, a2, b1, b2)]
        total[4:] += torch.stack([x.sum() for x in means])
    W, aa, bb, ab, a1, a2, b1, b2 = (total / draws).tolist()
    scale = N / (N - 1)
    return [scale * (aa / W - a1 / W * a2 / W), scale * (bb / W - b1 / W * b2 / W),
            scale * 0.5 * (ab / W - a1 / W * b2 / W - b1 / W * a2 / W)]


def _plug_in(w, psi, alpha, N):
    T = w.sum()
    a, b = (w * psi).sum() / T, (w * alpha).sum() / T
    return torch.stack([(w * psi * psi).sum() / T - a * a, (w * alpha * alpha).sum() / T - b * b,
                        (w * psi * alpha).sum() / T - a * b]) * (N / (N - 1))


def exact(case, seed):
    kind = case["kind"]
    if kind == "connected":             # whole numbers
        return None
    if kind == "batch":
        return [_Plain(p).fixed_effects() for p in _systems(case, seed)]
    if kind == "pass0":
        worker, fes, V, w = _raw(case, seed)
        cols = [torch.unique(c.long(), return_inverse=True) for c in (worker, *fes)]
        key = torch.zeros_like(cols[0][1])
        for u, c in cols:
            key = key * len(u) + c
        order = torch.argsort(key)
        return [cols[0][1][order].int(), torch.stack([c[order] for _, c in cols[1:]], 1).int(),
                V[order].T.contiguous(), None if w is None else w[order],
                [u.int() for u, _ in cols]]
    p = _panel(case, seed)
    if kind in ("fit", "fit_host"):
        return _Plain(p).fixed_effects()
    if kind == "solve":
        return _Plain(p).solve(*_right_sides(case, p))
    m = _Plain(p, covariates=kind != "estimate")
    if kind == "leverages":
        return list(_leverages(m, case["draws"], 11))
    beta, gam, alpha, e, V = m.regression()
    N, D = len(p.g), p.codes.shape[1]
    psi = gam[m.lev[0]]
    if kind == "kss":
        lev, com, factor = _leverages(m, case["draws"], 11)
        y = p.V[0]
        sigma2 = (y - y.mean()) * e / com * factor
        plug = _plug_in(m.w, psi, alpha[p.g], N).tolist()
        bias = _trace(m, sigma2, case["draws"], 11 + TRACE_SEED_OFFSET)
        return {"leverage": lev, "complement": com, "factor": factor, "sigma2": sigma2,
                "plug_in": plug, "bias": bias, "leave_out": [a - b for a, b in zip(plug, bias)]}
    if kind == "estimate":
        H, w = V[:, 1:], m.w
        k = H.shape[1]
        B = H.T @ (w[:, None] * H)
        s = (w * e)[:, None] * H
        rss, Binv = float((w * e * e).sum()), torch.linalg.inv(B)
        roots = m.components()
        # components of the pairs of dimensions: (workers, firms); the years
        # link everybody, so the pair with the most is the first
        parts = int((roots == torch.arange(len(roots), device=roots.device)).sum())
        k_fe = m.G + m.L - (parts + D - 1)
        out = {"beta": beta, "rss": rss, "k_fe": k_fe, "iid": rss / (N - k - k_fe) * Binv,
               "hetero": N / (N - k - k_fe) * Binv @ (s.T @ s) @ Binv}
        for name, idx, n in (("CRV1", p.g, m.G), ("CRV1:fe1", m.lev[0], p.n_levels[0])):
            S = m._sum(idx, s, n)
            adj = n / (n - 1) * (N - 1) / (N - (k + k_fe - n + 1))
            out[name] = adj * Binv @ (S.T @ S) @ Binv
        return out
    # adjoint: the gradient at theta, then one inverse and the row scatter
    th = [t.clone().requires_grad_(True) for t in (gam, alpha, m.w)]
    comp = _plug_in(th[2], th[0][m.lev[0]], th[1][p.g], N)
    out = {"beta": beta, "components": comp.detach()}
    d = torch.autograd.grad(comp[0], th, allow_unused=True)
    zero = [torch.zeros_like(t) for t in th]
    one = torch.zeros_like(beta)
    one[0] = 1.0
    for name, (dg, da, dw), db in (("var_psi", d, torch.zeros_like(beta)),
                                   ("beta0", zero, one)):
        da = torch.zeros_like(alpha) if da is None else da
        r = m.rows(*m.inverse(dg[:, None], db[:, None], da[:, None]))[:, 0]
        out[name] = [r * m.w] + ([r * e + dw] if p.w is not None else [])
    return out
