"""The calls that users of this framework make, as timed cases.

Each case is one pass through the public entry points (``api.Green``,
``api.CondOpt``, ``api.Batch``, ``api.pade_batch``): the model is set, solved
and its results are read back, as a program that scans models does.  Every
pass therefore sets its model anew; the solver contexts, which own the device
memory of every grid they have used, are kept for the whole program.

``exact`` restates the path in 64 bits with torch (dense DCT matrices, dense
spline solves, bracketed root searches), without the framework.
"""
import math

import numpy as np
import torch

from tpsc_conductivity_b200 import _lib, api

PI = math.pi
FORMS = {"fp64": _lib.FORM_REFERENCE, "newton": _lib.FORM_NEWTON, "mixed": _lib.FORM_NEWTON | _lib.FORM_MIXED}
# what a solve leaves in its scalars, the counts of evaluations apart
SOLVE = ("mu0", "chi0max", "Usp", "Uch", "dblOcc", "Sigma_inf", "mu", "trSG", "trSG_asymp", "trSG2", "dblOcc_SG2")
SCAN = api.Batch.CORR_COLUMNS


def listed():
    return [
        # one small lattice with the reference's root searches: a test or a
        # notebook cell, where launches and round trips count
        {"name": "solve_l16", "kind": "solve", "nk0": 16, "nw0": 64, "form": "fp64", "overlap": False},
        # the reference's driver program, stage by stage (half and full grid)
        {"name": "driver_l64", "kind": "driver", "nk0": 64, "nw0": 1024, "form": "fp64"},
        # the headline solve with Sigma(k, iw_n) streamed to the host beside the next solve
        {"name": "solve_l256_mixed", "kind": "solve", "nk0": 256, "nw0": 4096, "form": "mixed", "overlap": True},
        # optical conductivity with the Maki-Thompson correction, from the plain
        # FP64 lattice of the first examples to the headline size
        {"name": "cond_l32", "kind": "conductivity", "nk0": 32, "nw0": 512, "form": "fp64", "bins": 1, "nq": 16},
        {"name": "cond_l128_mixed", "kind": "conductivity", "nk0": 128, "nw0": 2048, "form": "mixed", "bins": 1,
         "nq": 256},
        {"name": "cond_l256", "kind": "conductivity", "nk0": 256, "nw0": 4096, "form": "newton", "bins": 3,
         "nq": 256},
        # sensitivities: the sum rules' forward tangents and sigma(iq_1)'s reverse pass
        {"name": "gradient_l128", "kind": "gradient", "nk0": 128, "nw0": 2048, "nq": 1},
        # the Aslamazov-Larkin correction, total and by angle
        {"name": "al_l32", "kind": "aslamazov_larkin", "nk0": 32, "nw0": 256, "mmin": 3, "bins": 1},
        {"name": "al_l64", "kind": "aslamazov_larkin", "nk0": 64, "nw0": 1024, "mmin": 4, "bins": 3},
        # many models of uneven lattices and cutoffs in one call
        {"name": "sweep_64", "kind": "sweep", "points": 64},
        # the reference's (density, temperature) scan of correlation lengths
        {"name": "scan_l64", "kind": "scan", "nk0": 64, "nw0": 512, "densities": 3, "temperatures": 5},
        # batched Pade continuation to the real axis
        {"name": "pade_153", "kind": "pade", "functions": 153, "nodes": 10, "energies": 1000},
    ]


def draw(rng):
    kind = rng.choice(["solve", "solve", "driver", "conductivity", "conductivity", "gradient", "aslamazov_larkin",
                       "sweep", "scan", "pade"])
    c = {"kind": kind}
    if kind == "solve":
        c.update(nk0=rng.choice([16, 32, 64, 128, 256]), nw0=rng.choice([64, 128, 256, 512, 1024, 2048, 4096]),
                 form=rng.choice(["fp64", "newton", "mixed"]), overlap=rng.choice([False, True]))
    elif kind == "driver":
        c.update(nk0=rng.choice([32, 64, 128]), nw0=rng.choice([128, 256, 512, 1024, 2048]), form="fp64")
    elif kind == "conductivity":
        c.update(nk0=rng.choice([16, 32, 64, 128, 256]), nw0=rng.choice([128, 256, 512, 1024, 2048, 4096]),
                 form=rng.choice(["fp64", "newton", "mixed"]), bins=rng.randint(1, 5))
        c["nq"] = rng.randint(1, c["nw0"] // 2)
    elif kind == "gradient":
        c.update(nk0=rng.choice([16, 32, 64, 128]), nw0=rng.choice([128, 256, 512, 1024, 2048]), nq=rng.randint(1, 32))
    elif kind == "aslamazov_larkin":
        c.update(nk0=rng.choice([16, 32, 64]), nw0=rng.choice([128, 256, 512]), mmin=rng.randint(2, 4),
                 bins=rng.randint(1, 5))
    elif kind == "sweep":
        c.update(points=int(round(math.exp(rng.uniform(math.log(5), math.log(64))))))
    elif kind == "scan":
        c.update(nk0=rng.choice([16, 32, 64]), nw0=rng.choice([128, 256, 512]), densities=rng.randint(1, 4),
                 temperatures=rng.randint(1, 6))
    else:
        c.update(functions=int(round(math.exp(rng.uniform(0, math.log(2145))))), nodes=rng.randint(4, 10),
                 energies=int(round(math.exp(rng.uniform(math.log(30), math.log(2000))))))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_kept = {}


def _handle(key, make):
    """The solver contexts a program keeps for all its calls."""
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _context(form):
    def make():
        ctx = api.Context()
        ctx.call("tpsc_set_form", FORMS[form])
        # a scan of models: each Newton-form solve is one graph launch, updated in place
        ctx.call("tpsc_set_graph_mode", 2)
        return ctx

    return _handle(form, make)


def _model(case, seed):
    """One model of the ranges of the named workloads: (n, T, (t', t'', t''', U))."""
    r = np.random.default_rng(seed)
    T = r.uniform(128.0, 256.0) / case["nw0"]
    if T > 0.5:
        T = r.uniform(0.25, 0.5)
    return (float(r.uniform(0.8, 0.95)), float(T),
            (float(r.uniform(-0.2, -0.05)), float(r.uniform(-0.05, 0.05)), 0.0, float(r.uniform(2.0, 4.0))))


def _points(case, seed):
    """Rows (nk0, Nw0, n, T, t', t'', t''', U) of the parameter sweep."""
    r = np.random.default_rng(seed)
    p = np.zeros((case["points"], 8))
    for row in p:
        T = math.exp(r.uniform(math.log(0.03), math.log(0.5)))
        nw0 = 2 * 2 ** math.ceil(math.log2(math.ceil(40.0 / (PI * T))))
        row[:] = (r.choice([32, 64, 128, 256]), nw0, r.uniform(0.7, 1.0), T, r.uniform(-0.3, 0.0), 0.0, 0.0,
                  r.uniform(1.0, 6.0))
    return p


def _scan(case, seed):
    r = np.random.default_rng(seed)
    dens = np.sort(r.uniform(0.75, 0.95, 2))  # the first and the last of the scan
    temp = np.sort(r.uniform(128.0, 256.0, 2) / case["nw0"])[::-1].copy()
    return (float(r.uniform(-0.2, -0.05)), 0.0, 0.0, float(r.uniform(2.0, 3.0))), dens, temp


def _pade(case, seed):
    """Matsubara samples of functions with continuous spectra (semicircles of
    drawn centres and widths) and the energies to continue them to."""
    r = np.random.default_rng(seed)
    nf, nn, nz = case["functions"], case["nodes"], case["energies"]
    x = 1j * (2 * np.arange(nn) + 1) * PI * 0.25
    c, w = r.uniform(-2.0, 2.0, (nf, 1)), r.uniform(1.5, 4.0, (nf, 1))
    z = x[None, :] - c
    y = 2.0 * (z - 1j * np.sqrt(w * w - z * z)) / (w * w)
    return np.broadcast_to(x, (nf, nn)).copy(), y, np.linspace(-8.0, 8.0, nz) + 0.05j


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "sweep":
        s["points"] = _points(case, seed)
        s["batch"] = _handle("batch", api.Batch)
        s["batch"].set_graph_mode(3)
    elif kind == "scan":
        s["scan"] = _scan(case, seed)
        s["batch"] = _handle("scan batch", api.Batch)
    elif kind == "pade":
        s["pade"] = _pade(case, seed)
        s["ctx"] = _context("fp64")
    else:
        s["model"] = _model(case, seed)
        s["ctx"] = _context(case.get("form", "newton"))
        if kind in ("solve", "driver"):
            nbk = case["nk0"] // 2 + 1
            out = torch.empty((case["nw0"] // 2, nbk * (nbk + 1) // 2), dtype=torch.complex64, pin_memory=True)
            s["sigma"] = out.numpy()
    return s


def _as_form(case, v):
    """Results in the precision that the form states: the mixed form's single."""
    v = np.asarray(v)
    return v.astype(np.float32) if case.get("form") == "mixed" and v.dtype == np.float64 else v


def _solved(case, sc):
    return _as_form(case, [sc[k] for k in SOLVE])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sweep":
        res, status, _ = state["batch"].solve(state["points"])
        cols = [_lib.SCALARS.index(k) for k in SOLVE]
        return {"scalars": res[:, cols].astype(np.float32), "status": status}
    if kind == "scan":
        params, dens, temp = state["scan"]
        rows, status, _ = state["batch"].corr_length(case["nk0"], case["nw0"], params, dens, case["densities"], temp,
                                                     case["temperatures"])
        return {"rows": {k: rows[:, i] for i, k in enumerate(SCAN)}, "status": status}
    if kind == "pade":
        return api.pade_batch(*state["pade"], ctx=state["ctx"])
    n, T, params = state["model"]
    if kind in ("solve", "driver"):
        g = api.Green(case["nk0"], case["nw0"], n, T, 0.1, params, ctx=state["ctx"])
        if kind == "solve":
            g.solve()
            g.sigma_async32(state["sigma"])
            if not case["overlap"]:
                g.wait_copies()
            return {"scalars": _solved(case, g.scalars()), "sigma": state["sigma"]}
        g.calc_Self_FFT_spline()
        g.traceSelfG()
        g.find_mu()
        g.sigma_async32(state["sigma"])
        g.wait_copies()
        sc = g.scalars()
        return {"scalars": _solved(case, sc), "difference": np.array([sc["difRelsp"], sc["difRelch"]]),
                "sigma": state["sigma"]}
    g = api.CondOpt(case["nk0"], case["nw0"], n, T, 0.1, params, ctx=state["ctx"])
    g.solve()
    if kind == "gradient":
        tangents = g.sumrule_tangents()
        cot = np.zeros(case["nq"])
        cot[-1] = 1.0
        grad, dD = g.sigma_qn_vjp(cot)
        return {"sum_rules": np.array([[tangents[p][k] for k in ("Usp", "Uch", "D")] for p in ("U", "mu", "tp")]),
                "grad": grad, "dD": dD}
    if kind == "aslamazov_larkin":
        r = g.calc_chijj_vertex_corr_all_optim(True, case["mmin"], case["bins"])
        return {k: np.asarray(r[k]) for k in ("chijj1", "chijj2", "kx0", "ind_freq", "chijj3", "chijj3_k")}
    r = g.calc_chijj_vertex_corr_all_optim(N_theta_k=case["bins"])
    sigma, bubble = g.sigma_qn(case["nq"])
    out = {k: r[k] for k in ("chijj1", "chijj2", "kx0", "chijj1_k", "chijj2_k")}
    out.update(sigma=sigma, bubble=bubble, scalars=_solved(case, g.scalars()))
    return {k: _as_form(case, v) for k, v in out.items()}


# ---------------------------------------------------------------------------
# the work that a pass cannot do without
# ---------------------------------------------------------------------------
def _fft(n):
    """A real-even transform of n points."""
    return 1.25 * n * max(1.0, math.log2(n))


def _solve_work(nk0, nw0):
    """Slices of G, chi0 (half of tau), V (half) and Sigma, then the tau
    transforms of chi0, V and Sigma, the sums over chi0 and Sigma."""
    nbk, n8 = nk0 // 2 + 1, (nk0 // 2 + 1) * (nk0 // 2 + 2) // 2
    slices = 3 * nw0 * 2 * nbk * _fft(nk0)
    tau = n8 * (2 * _fft(nw0) + 2 * _fft(nw0) + 10 * 2 * nw0)
    return slices + tau + n8 * nw0 * 20


def _cond_work(nk0, nw0):
    """The h and f0 slices there and back, six transforms and four splines along tau."""
    nbk = nk0 // 2 + 1
    k4 = (nbk - 2) * nbk
    return 2 * nw0 * 2 * 2 * nbk * _fft(nk0) + k4 * (6 * 2 * _fft(nw0) + 60 * nw0)


def work(case):
    kind = case["kind"]
    if kind == "sweep":
        p = _points(case, 0)
        return {"bytes": 8.0 * case["points"] * (8 + len(SOLVE)), "flops": sum(_solve_work(r[0], r[1]) for r in p)}
    if kind == "scan":
        n = case["densities"] * case["temperatures"]
        one = _solve_work(case["nk0"], case["nw0"]) / 3 * 1.125
        return {"bytes": 8.0 * n * (2 + len(SCAN)), "flops": n * one}
    if kind == "pade":
        f, m, z = case["functions"], case["nodes"], case["energies"]
        return {"bytes": 16.0 * (2 * f * m + z + f * z), "flops": 30.0 * f * m * (m / 2 + 3 * z)}
    nk0, nw0 = case["nk0"], case["nw0"]
    n8, k4 = (nk0 // 2 + 1) * (nk0 // 2 + 2) // 2, (nk0 // 2 - 1) * (nk0 // 2 + 1)
    if kind in ("solve", "driver"):
        more = 1.125 if kind == "driver" else 1.0
        return {"bytes": 8.0 * n8 * nw0 / 2 + 8.0 * 19, "flops": more * _solve_work(nk0, nw0)}
    flops = _solve_work(nk0, nw0) + _cond_work(nk0, nw0)
    size = 8.0 * (8 + 4 * (nw0 // 2 + 1))
    if kind == "gradient":
        flops = 3 * flops
    if kind == "aslamazov_larkin":
        m = case["mmin"]
        freqs = (nw0 // 2 >> m) + m * (nw0 // 2 >> (m + 1))
        flops += freqs * (6 * nw0 * 2 * (nk0 // 2 + 1) * _fft(nk0) + k4 * nw0 * (12 * math.log2(nw0) + 100))
    return {"bytes": size, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _t(v):
    return torch.as_tensor(v, dtype=torch.float64, device="cuda")


def _root(f, lo, hi):
    """Zero of f in [lo, hi] by Ridders' method, to the last bits."""
    a, b = lo, hi
    fa, fb = f(a), f(b)
    for _ in range(200):
        m = 0.5 * (a + b)
        fm = f(m)
        if fm == 0.0:
            return m
        d = math.sqrt(max(fm * fm - fa * fb, 0.0))
        x = m + (m - a) * (1.0 if fa >= fb else -1.0) * fm / d if d else m
        fx = f(x)
        if fx == 0.0:
            return x
        if fm * fx < 0:
            a, fa, b, fb = (m, fm, x, fx) if m < x else (x, fx, m, fm)
        elif fa * fx < 0:
            b, fb = x, fx
        else:
            a, fa = x, fx
        if b - a <= 4e-16 * max(1.0, abs(a)):
            break
    return a if abs(fa) < abs(fb) else b


def _spline(V, h, d0, dN):
    """Second derivatives at the nodes of the clamped cubic spline (axis 0)."""
    n = V.shape[0]
    one = torch.ones(n - 1, dtype=torch.float64, device="cuda")
    A = 4.0 * torch.eye(n, dtype=torch.float64, device="cuda") + torch.diag(one, 1) + torch.diag(one, -1)
    A[0, 0] = A[n - 1, n - 1] = 2.0
    rhs = torch.empty_like(V)
    rhs[1:-1] = 6.0 / (h * h) * (V[2:] - 2.0 * V[1:-1] + V[:-2])
    rhs[0] = 6.0 / h * ((V[1] - V[0]) / h - d0)
    rhs[-1] = 6.0 / h * (dN - (V[-1] - V[-2]) / h)
    return torch.linalg.solve(A, rhs)


def _integral(V, M, h):
    """Integral of the spline over its nodes."""
    return h * (V.sum(0) - 0.5 * (V[0] + V[-1])) - h ** 3 / 24.0 * (2.0 * M.sum(0) - M[0] - M[-1])


class _Lattice:
    """Tables of one lattice: octant points m + l (l+1)/2, their weights (the
    zone's points per octant point) and the DCT-I and DST-I matrices."""

    def __init__(self, nk0):
        self.L, self.nbk = nk0, nk0 // 2 + 1
        N = self.nbk - 1
        i = torch.arange(self.nbk, device="cuda")
        self.cos = torch.cos(PI * i.double() / N)
        self.dct = 2.0 * torch.cos(PI * ((i[:, None] * i[None, :]) % (2 * N)).double() / N)
        self.dct[:, 0] *= 0.5
        self.dct[:, N] *= 0.5
        j = torch.arange(1, N, device="cuda")
        self.dst = 2.0 * torch.sin(PI * ((j[:, None] * j[None, :]) % (2 * N)).double() / N)
        self.l, self.m = torch.tril_indices(self.nbk, self.nbk, device="cuda")
        edge = torch.where((i == 0) | (i == N), 1.0, 2.0).double()
        self.w = edge[self.l] * edge[self.m] * torch.where(self.l == self.m, 1.0, 2.0)
        # the interior kx points (l + 1, m) of the current vertex, and their octant points
        x, y = j[:, None].expand(N - 1, self.nbk), i[None, :].expand(N - 1, self.nbk)
        hi, lo = torch.maximum(x, y), torch.minimum(x, y)
        self.k4 = (lo + hi * (hi + 1) // 2).reshape(-1)
        self.wt = torch.where((y == 0) | (y == N), 2.0, 4.0).double().reshape(-1)
        self.x4, self.y4 = x.reshape(-1), y.reshape(-1)

    def octant(self, a):
        """DCT-I x DCT-I of octant arrays [..., n8]."""
        flat = a.reshape(-1, a.shape[-1])
        out = torch.empty_like(flat)
        for s in range(0, flat.shape[0], 512):
            full = torch.empty((min(512, flat.shape[0] - s), self.nbk, self.nbk), dtype=torch.float64, device="cuda")
            full[:, self.l, self.m] = flat[s:s + 512]
            full[:, self.m, self.l] = flat[s:s + 512]
            out[s:s + 512] = (self.dct @ full @ self.dct.T)[:, self.l, self.m]
        return out.reshape(a.shape)

    def interior(self, a):
        """DST-I x DCT-I of arrays [..., K4]."""
        if a.is_complex():
            return torch.complex(self.interior(a.real.contiguous()), self.interior(a.imag.contiguous()))
        flat = a.reshape(-1, self.nbk - 2, self.nbk)
        out = torch.empty_like(flat)
        for s in range(0, flat.shape[0], 512):
            out[s:s + 512] = self.dst @ flat[s:s + 512] @ self.dct.T
        return out.reshape(a.shape)


class _Solve:
    """chi0 -> Usp, Uch -> V -> Sigma -> mu of one model."""

    def __init__(self, nk0, nw0, n, T, params, mu_shift=0.0, stop="mu"):
        lat = self.lat = _handle(("lattice", nk0), lambda: _Lattice(nk0))
        tp, tpp, t3, U = params
        self.n, self.T, self.U, self.nw0, self.params = n, T, U, nw0, params
        w, L2, beta = lat.w, float(nk0 * nk0), 1.0 / T
        c1 = lat.cos
        c2 = torch.cos(2.0 * PI * torch.arange(lat.nbk, device="cuda").double() / (lat.nbk - 1))
        l, m = lat.l, lat.m
        self.e = e = (-2.0 * (c1[l] + c1[m]) - 4.0 * tp * c1[l] * c1[m] - 2.0 * tpp * (c2[l] + c2[m])
                      - 4.0 * t3 * (c2[l] * c1[m] + c2[m] * c1[l]))
        self.mu0 = mu_shift
        if not (n == 1.0 and tp == 0 and tpp == 0):
            self.mu0 += _root(lambda x: float((2.0 * w / (torch.exp((e - x) / T) + 1.0)).sum()) / L2 - n, -8.0, 8.0)
        x = self.x = e - self.mu0
        er = torch.zeros_like(e)
        er[1:5] = _t([-1.0, -tp, -tpp, -t3])
        nb = nw0 // 2 + 1
        h = self.h = 1.0 / (nw0 * T)

        # G(r, tau) and the tau-derivatives at its ends
        def g0(t):
            return torch.where(x > 0, -torch.exp(-t * x) / (torch.exp(-x / T) + 1.0),
                               -torch.exp((beta - t) * x) / (torch.exp(x / T) + 1.0)) / L2

        tau = _t(np.arange(nw0 + 1)) * h
        G = self.G = lat.octant(g0(tau[:, None]))
        self.dGp = lat.octant(-x * g0(0.0))
        delta = torch.zeros_like(e)
        delta[0] = 1.0
        self.dGm = er - self.mu0 * delta - self.dGp
        chirt = torch.empty((nb, e.numel()), dtype=torch.float64, device="cuda")
        chirt[1:] = -2.0 * G[1:nb] * -G[nw0 - torch.arange(1, nb, device="cuda")]
        chirt[0] = -2.0 * G[0] * (G[0] + delta)
        self.dchi = -2.0 * (self.dGp * (G[0] + delta) + self.dGm * G[0])
        slope = lat.octant(self.dchi)
        chiqt = lat.octant(chirt)
        M = _spline(chiqt, h, slope, torch.zeros_like(slope))
        f = torch.cat([(M[1:] - M[:-1]) / h, -((M[1:] - M[:-1]) / h).flip(0)])
        F = torch.fft.ifft(f, dim=0) * nw0
        j = _t(np.arange(1, nb))[:, None]
        wn, th = 2.0 * j * PI * T, 2.0 * j * PI / nw0
        chi = self.chi = torch.empty_like(chirt)
        chi[0] = 2.0 * _integral(chiqt, M, h)
        chi[1:] = -2.0 * slope / wn ** 2 + ((1.0 - torch.cos(th)) * F[1:nb].real + torch.sin(th) * F[1:nb].imag) / wn ** 4
        chi[1:, 0] = 0.0
        self.ci, self.ci2 = -2.0 * slope, 2.0 * F[nb - 1].real.clone()
        self.ci[0] = self.ci2[0] = 0.0
        self.chi0max = float(chi[0].max())

        # the sum rules
        wt = _t(np.arange(nb, nw0 + 1))[:, None] * 2.0 * PI * T
        tail = self.ci / wt ** 2 + self.ci2 / wt ** 4
        wj = torch.full((nb, 1), 1.0, dtype=torch.float64, device="cuda")
        wj[0] = 0.5

        def trace(s):
            return 2.0 * T / L2 * float((wj * w * (chi / (1.0 + s * chi / 2.0) - chi)).sum()
                                        + (w * (tail / (1.0 + s * tail / 2.0) - tail)).sum())

        nsr = 2.0 - n if n > 1.0 else n
        base = n - n * n / 2.0
        self.Usp = _root(lambda u: trace(-u) + base - nsr + u * nsr * nsr / (2.0 * U), 0.0,
                         2.0 / self.chi0max * (1.0 - 1e-13))
        self.Uch = _root(lambda u: trace(u) + base - nsr - self.Usp * nsr * nsr / (2.0 * U) + nsr * nsr, 0.0, 1000.0 * U)
        self.D = self.Usp / U * nsr * nsr / 4.0 + (1.0 - nsr if n > 1.0 else 0.0)
        if stop == "roots":
            return
        Usp, Uch = self.Usp, self.Uch

        # V(r, tau), Sigma(k, tau)
        vq = T / L2 * U * (3.0 * Usp * (chi / (1.0 - Usp * chi / 2.0) - chi)
                           + Uch * (chi / (1.0 + Uch * chi / 2.0) - chi)) / 8.0
        i = torch.arange(nb, device="cuda")
        D1 = 2.0 * torch.cos(PI * ((i[:, None] * i[None, :]) % nw0).double() * 2.0 / nw0)
        D1[:, 0] *= 0.5
        D1[:, nb - 1] *= 0.5
        fact = U * (3.0 * Usp + Uch) / 8.0
        V = self.V = D1 @ lat.octant(vq) + fact * chirt
        del D1
        tauv = torch.minimum(torch.arange(nw0 + 1, device="cuda"), nw0 - torch.arange(nw0 + 1, device="cuda"))
        st = lat.octant(G * V[tauv])
        gb = -(delta + G[0])
        d0 = lat.octant(fact * self.dchi * G[0] + V[0] * self.dGp)
        dN = lat.octant(-fact * self.dchi * gb + V[0] * self.dGm)
        M = _spline(st, h, d0, dN)
        k = _t(np.arange(nw0))[:, None]
        F = torch.fft.ifft(torch.exp(1j * k * PI / nw0) * (M[1:] - M[:-1]) / h, dim=0)[:nw0 // 2] * nw0
        k = k[:nw0 // 2]
        S = (1.0 - torch.exp(1j * (2.0 * k + 1.0) * PI / nw0)) * F
        self.Sinf = -float(st[0, 0] + st[nw0, 0])
        self.S2, self.S3, self.S4, self.S = d0 + dN, -(M[0] + M[-1]), S[-1].real.clone(), S
        z = self.z = 1j * (2.0 * k + 1.0) * PI * T
        sig = self.sigma = self.Sinf / z + self.S2 / z ** 2 + self.S3 / z ** 3 + S / z ** 4

        # the traces and mu
        wn = z.imag
        d = wn * wn + x * x
        self.trSG = float((2.0 * w * T / L2 / d * (-sig.real * x + sig.imag * wn)).sum())
        big = x.abs() > 1e-12
        ex = torch.exp(-x.abs() / T)
        a = torch.where(big, (1.0 / (torch.exp(x / T) + 1.0) - 0.5) / torch.where(big, x, torch.ones_like(x)),
                        -ex / ((ex + 1.0) ** 2 * T))
        self.trSGa = self.trSG + self.Sinf / L2 * float((w * (2.0 * T / d).sum(0) + w * a).sum())
        wl = _t(np.arange(nw0 // 2, nw0 + 1))[:, None] * 2.0 * PI * T + PI * T
        zl = torch.complex(-self.S2 / wl ** 2 + self.S4 / wl ** 4, wl * 0 + (-self.Sinf / wl + self.S3 / wl ** 3))
        zs, zt = z - x - self.mu0 - sig, 1j * wl - x - self.mu0 - zl
        g00, g0t = 1.0 / (z - x), 1.0 / (1j * wl - x)

        def diff(p):
            one = (sig - (p - self.mu0)) / (zs + p) * g00
            two = (zl - (p - self.mu0)) / (zt + p) * g0t
            return float((2.0 * w * one.real).sum() + (2.0 * w * two.real).sum())

        self.mu = _root(diff, -10.0, 10.0)
        gm = 1.0 / (zs + self.mu)
        self.trSG2 = 2.0 * T / L2 * float((w * (sig * gm).real).sum())

    def scalars(self):
        return np.array([self.mu0, self.chi0max, self.Usp, self.Uch, self.D, self.Sinf, self.mu, self.trSG, self.trSGa,
                         self.trSG2, (self.trSG2 + self.U * self.n * self.n / 4.0) / self.U])


def _velocity(s):
    """d eps/d kx on the interior points, d2 eps/d kx2 there and on the kx = 0, pi lines."""
    lat = s.lat
    tp, tpp, t3, _ = s.params
    N = lat.nbk - 1

    def dk(kx, ky):
        return (2.0 * torch.sin(kx) + 4.0 * tp * torch.sin(kx) * torch.cos(ky) + 4.0 * tpp * torch.sin(2 * kx)
                + 4.0 * t3 * (2.0 * torch.sin(2 * kx) * torch.cos(ky) + torch.cos(2 * ky) * torch.sin(kx)))

    def d2k(kx, ky):
        return (2.0 * torch.cos(kx) + 4.0 * tp * torch.cos(kx) * torch.cos(ky) + 8.0 * tpp * torch.cos(2 * kx)
                + 4.0 * t3 * (4.0 * torch.cos(2 * kx) * torch.cos(ky) + torch.cos(2 * ky) * torch.cos(kx)))

    kx, ky = lat.x4.double() * PI / N, lat.y4.double() * PI / N
    y = torch.arange(lat.nbk, device="cuda").double() * PI / N
    return dk(kx, ky), d2k(kx, ky), [d2k(0.0 * y, y), d2k(0.0 * y + PI, y)]


def _bins(s, nbins):
    lat = s.lat
    th = torch.atan((lat.L / 2 - lat.y4.double()) / (lat.L / 2 - lat.x4.double()))
    return torch.floor(th / (PI / (2.0 * nbins))).long().clamp(0, nbins - 1)


def _conductivity(s, nbins=1):
    """chi_jj's bubble and Maki-Thompson parts, per angle and in all, and kx0."""
    lat, T, nw0, h, mu = s.lat, s.T, s.nw0, s.h, s.mu
    L2, beta, no = float(lat.L ** 2), 1.0 / s.T, s.nw0 // 2
    dk, d2k, lines = _velocity(s)
    x, e = s.x[lat.k4], s.e[lat.k4]
    tau = _t(np.arange(nw0 + 1))[:, None] * h
    fold = torch.minimum(torch.arange(nw0 + 1, device="cuda"), nw0 - torch.arange(nw0 + 1, device="cuda"))
    f = 1.0 / (torch.exp(x / T) + 1.0)
    low, a = x <= 0, dk / L2
    # h = a exp(-x tau) (1 - f), f0 = (tau - beta f) h, in the stable form of each sign
    decay = torch.where(low, torch.exp(x * (beta - tau)) * f, torch.exp(-x * tau) * (1.0 - f))

    def to_k(v, dv0, dvb):
        v, dv0, dvb = lat.interior(v), lat.interior(dv0), lat.interior(dvb)
        fact = s.U * (3.0 * s.Usp + s.Uch) / 4.0
        dchi, V0 = s.dchi[lat.k4], s.V[0][lat.k4]
        d0 = lat.interior(2.0 * dv0 * V0 + v[0] * fact * dchi)
        db = lat.interior(2.0 * dvb * V0 - v[nw0] * fact * dchi)
        return lat.interior(2.0 * v * s.V[fold][:, lat.k4]), d0, db

    k = _t(np.arange(nw0))[:, None]
    kn = (2.0 * (k - no) + 1.0) * PI * T  # both signs

    def fermionic(v, d0, db):
        M = _spline(v, h, d0, db)
        F = torch.fft.ifft(torch.exp(1j * k * PI / nw0) * (M[1:] - M[:-1]) / h, dim=0) * nw0
        F = torch.roll(F, no, 0)
        C1, C2, C3 = -v[0] - v[nw0], d0 + db, -(M[0] + M[-1])
        ph = 1.0 - torch.exp(1j * (2.0 * (k - no) + 1.0) * PI / nw0)
        return -1j * C1 / kn - C2 / kn ** 2 + 1j * C3 / kn ** 3 + ph * F / kn ** 4, C1

    hv = a * decay
    J, C1 = fermionic(*to_k(hv, -x * hv[0], -x * hv[nw0]))
    f0 = hv * (tau - beta * f)
    J0, _ = fermionic(*to_k(f0, hv[0] - x * f0[0], hv[nw0] - x * f0[nw0]))
    sig = torch.cat([s.sigma.flip(0).conj(), s.sigma])
    G = T / (1j * kn - e + mu - sig[:, lat.k4])
    J = G * J
    q0 = (G * G * J0 / T).sum(0).real
    del J0
    tail = T / (mu - e + 1j * (kn + s.Sinf / kn))
    G = G - tail
    J = J - tail * (-1j * C1 / kn)
    del tail

    def split(e):
        r = torch.sqrt((mu - e) ** 2 + 4.0 * s.Sinf)
        r1 = torch.where(mu - e >= 0, 0.5 * (-(mu - e) - r), -2.0 * s.Sinf / (-(mu - e) + r))
        return r1, -s.Sinf / r1  # the negative and the positive root

    def fermi(r):
        return 1.0 / (torch.exp(-r.abs() / T) + 1.0), torch.exp(-r.abs() / T) / (torch.exp(-r.abs() / T) + 1.0)

    r1, r2 = split(e)
    big1, sml1 = fermi(r1)
    big2, sml2 = fermi(r2)
    a1, a2, b1 = r1 / (r1 - r2), r2 / (r2 - r1), C1 / (r1 - r2)
    k0 = G.sum(0).real + a1 * big1 + a2 * sml2
    dG, dJ = (kn * G.imag).sum(0), (kn * J.imag).sum(0)
    dGp, dGm = dG + r1 * a1 * sml1 + r2 * a2 * big2, -dG + r1 * a1 * big1 + r2 * a2 * sml2
    dJ0, dJb = -dJ + r1 * b1 * big1 - r2 * b1 * sml2, dJ + r1 * b1 * sml1 - r2 * b1 * big2
    t = tau[:nw0]
    Gt = (torch.exp(1j * k * PI * (nw0 - 1) / nw0) * torch.fft.fft(G, dim=0)).real
    Gt -= a1 * torch.exp((beta - t) * r1) * big1 + a2 * torch.exp(-t * r2) * big2
    del G
    raw = torch.exp(-1j * k * PI * (nw0 - 1) / nw0) * torch.fft.ifft(J, dim=0) * nw0
    Jt = raw.real + b1 * torch.exp(t * r1) * big1 - b1 * torch.exp((t - beta) * r2) * big2
    Jb = -raw[0].real + b1 * sml1 - b1 * big2
    del J, raw
    gj = torch.cat([Gt * Jt, ((-Gt[0] - 1.0) * Jb)[None]])
    M = _spline(gj, h, dGp * Jt[0] + Gt[0] * dJ0, dGm * Jb - (Gt[0] + 1.0) * dJb)
    F = torch.fft.fft((M[1:] - M[:-1]) / h, dim=0)[1:no + 1]
    q = _t(np.arange(1, no + 1))[:, None]
    wq = 2.0 * q * PI * T
    ph = 1.0 - torch.exp(-2j * q * PI / nw0)
    Jq = -2.0 * (gj[0] - gj[nw0]) / wq + 2.0 * (M[0] - M[-1]) / wq ** 3 + 2.0 * (ph * F).imag / wq ** 4
    del gj, Jt
    gg = torch.cat([(Gt[0] * (Gt[0] + 1.0))[None], -Gt[1:no + 1] * Gt[nw0 - torch.arange(1, no + 1, device="cuda")]])
    dchi = dGp * (Gt[0] + 1.0) + Gt[0] * dGm
    M = _spline(gg, h, dchi, torch.zeros_like(dchi))
    A = (M[1:] - M[:-1]) / h
    F = torch.fft.fft(torch.cat([A, -A.flip(0)]), dim=0)[1:no + 1]
    bub = torch.cat([2.0 * _integral(gg, M, h)[None], -2.0 * dchi / wq ** 2 + (ph * F).real / wq ** 4])
    c1 = -2.0 * lat.wt / L2 * dk * dk * bub
    c2 = -lat.wt / L2 * dk * torch.cat([q0[None], Jq / wq])
    bins = _bins(s, nbins)
    per = [torch.stack([c[:, bins == b].sum(1) for b in range(nbins)], 1) for c in (c1, c2)]
    kx0 = -float((2.0 * lat.wt / L2 * d2k * k0).sum())
    for l, d2 in zip((0, lat.nbk - 1), lines):
        y = torch.arange(lat.nbk, device="cuda")
        o = (y if l else 0 * y) + (torch.maximum(y, 0 * y + l) * (torch.maximum(y, 0 * y + l) + 1)) // 2
        el = s.e[o]
        g = T / (1j * kn - el + mu - sig[:, o]) - T / (mu - el + 1j * (kn + s.Sinf / kn))
        p1, p2 = split(el)
        kk = g.sum(0).real + p1 / (p1 - p2) * fermi(p1)[0] + p2 / (p2 - p1) * fermi(p2)[1]
        wl = torch.where((y == 0) | (y == lat.nbk - 1), 1.0, 2.0)
        kx0 -= float((2.0 * wl / L2 * d2 * kk).sum())
    c1, c2 = c1.sum(1), c2.sum(1)
    wq = wq[:, 0]
    return {"chijj1": c1, "chijj2": c2, "kx0": np.asarray(kx0), "chijj1_k": per[0], "chijj2_k": per[1],
            "sigma": (-kx0 - c1[1:] - c2[1:]) / wq, "bubble": (-kx0 - c1[1:]) / wq}


def _aslamazov_larkin(s, mmin, nbins):
    """chi_jj's Aslamazov-Larkin part on the non-uniform frequency grid."""
    lat, T, nw0, h, mu, U = s.lat, s.T, s.nw0, s.h, s.mu, s.U
    L2, beta, no = float(lat.L ** 2), 1.0 / s.T, s.nw0 // 2
    dk, _, _ = _velocity(s)
    x, e, o = s.x[lat.k4], s.e[lat.k4], lat.k4
    f = 1.0 / (torch.exp(x / T) + 1.0)
    tau = _t(np.arange(nw0 + 1))[:, None] * h
    hk = dk / L2 * torch.where(x <= 0, torch.exp(x * (beta - tau)) * f, torch.exp(-x * tau) * (1.0 - f))
    Gm = -s.G.flip(0)[:, o]  # G(r, -tau)
    dg0, dgb = s.dGm[o], s.dGp[o]
    hr, d0, db = lat.interior(hk), lat.interior(-x * hk[0]), lat.interior(-x * hk[nw0])
    s0, sb = lat.interior(d0 * Gm[0] + hr[0] * dg0), lat.interior(db * Gm[nw0] + hr[nw0] * dgb)
    hg = lat.interior(hr * Gm)
    M = _spline(hg, h, s0, sb)
    F = torch.fft.fft((M[1:] - M[:-1]) / h, dim=0)
    p = _t(np.arange(no))[:, None]
    hq = 2.0 * ((1.0 - torch.exp(-2j * p * PI / nw0)) * F[:no]).real
    hq0, hg2 = 2.0 * _integral(hg, M, h), 2.0 * (s0 - sb)
    ci, ci2, chi = s.ci[o], s.ci2[o], s.chi[:, o]

    def chi_at(p):
        p = p.abs()
        wn = 2.0 * PI * T * p.clamp(min=1).double()[:, None]
        return torch.where((p <= no)[:, None], chi[p.clamp(max=no)], ci / wn ** 2 + ci2 / wn ** 4)

    def hg_at(p):
        p = p.abs()
        wn = 2.0 * PI * T * p.clamp(min=1).double()[:, None]
        return torch.where((p == 0)[:, None], hq0, -hg2 / wn ** 2 + hq[p.clamp(max=no - 1)] / wn ** 4)

    def quotient(p1, p2):
        return (hg_at(p1) - hg_at(p2)) / (chi_at(p1) - chi_at(p2))

    jf, nj = no >> mmin, no >> (mmin + 1)
    grid, d = list(range(jf + 1)), 1
    for _ in range(mmin):
        d *= 2
        grid += [grid[-1] + d * (i + 1) for i in range(nj)]
    zs, zc = 1j * torch.sqrt(s.Usp * ci / 2.0), torch.sqrt(s.Uch * ci / 2.0)
    j = torch.arange(nw0, device="cuda")
    wt, bins = lat.wt, _bins(s, nbins)
    c3, c3k = np.zeros(len(grid)), np.zeros((len(grid), nbins))
    S = torch.cat([s.S.flip(0).conj(), s.S])[:, o]
    S2, S3 = s.S2[o], s.S3[o]
    # the asymptote's closed form in tau, and its derivatives at the ends
    e0, e1 = torch.exp(-zs * beta) - 1.0, torch.exp(zs * beta) - 1.0
    ec = torch.exp(-zc * beta)
    tsp = torch.exp(-zs * tau) / (e0 * 2.0 * zs) - torch.exp(zs * tau) / (e1 * 2.0 * zs)
    tch = torch.exp(-zc * tau) / ((ec - 1.0) * 2.0 * zc) - torch.exp(-zc * (beta - tau)) / ((1.0 - ec) * 2.0 * zc)
    shape = hg2 * (3.0 * s.Usp * tsp + s.Uch * tch)
    ends = []
    for t in (0.0, beta):
        dsp = -0.5 * torch.exp(-zs * t) / e0 - 0.5 * torch.exp(zs * t) / e1
        dch = -0.5 * torch.exp(-zc * t) / (ec - 1.0) - 0.5 * torch.exp(-zc * (beta - t)) / (1.0 - ec)
        ends.append(hg2 * (3.0 * s.Usp * dsp + s.Uch * dch))

    def to_matsubara(v, d0, db):
        M = torch.complex(_spline(v.real.contiguous(), h, d0.real, db.real),
                          _spline(v.imag.contiguous(), h, d0.imag, db.imag))
        ph = torch.exp(-1j * PI * j.double() / nw0)[:, None]
        F = torch.fft.fft(ph * (M[1:] - M[:-1]) / h, dim=0)

        def at(f, has, at):
            f = f.double()
            w = ((2.0 * f + 1.0) * PI * T)[:, None]
            out = -1j * (v[0] + v[nw0]) / w - (d0 + db) / w ** 2 + 1j * (M[0] + M[-1]) / w ** 3
            ph = 1.0 - torch.exp(-1j * (2.0 * f + 1.0) * PI / nw0)[:, None]
            return out + torch.where(has[:, None], ph * F[at] / w ** 4, 0.0)

        return at

    def green(f):
        w = ((2.0 * f.double() + 1.0) * PI * T)[:, None]
        has = ((f >= -no) & (f < no))[:, None]
        sg = -S2 / w ** 2 + 1j * (-s.Sinf / w + S3 / w ** 3) + torch.where(has, S[(f + no).clamp(0, nw0 - 1)] / w ** 4, 0.0)
        return 1.0 / (1j * w - e + mu - sg)

    for n in range(1, len(grid)):
        nn = grid[n]
        p1 = torch.where(j < no - nn // 2, j, j - nw0)
        p2 = p1 + nn
        D = quotient(p1, p2)
        if nn % 2 == 0:
            one = torch.tensor([-(nn // 2)], device="cuda")
            D[nw0 - nn // 2] = ((4.0 * quotient(one - 1, one - 1 + nn) - quotient(one - 2, one - 2 + nn)) / 3.0)[0]
        c = chi_at(p1)
        w = 2.0 * PI * T * p1.double()[:, None]
        hinf = hg2 * (3.0 * s.Usp / (-w * w + s.Usp * ci / 2.0) + s.Uch / (-w * w - s.Uch * ci / 2.0))
        ft = T * ((3.0 * s.Usp * c / (1.0 - s.Usp * c / 2.0) + s.Uch * c / (1.0 + s.Uch * c / 2.0)) * D - hinf)
        dt0 = -(w * ft).sum(0)
        ft = torch.fft.fft(ft, dim=0)
        H = lat.interior((torch.cat([ft, ft[:1]]) + shape) / L2)
        dH = [lat.interior((1j * dt0 + v) / L2) for v in ends]
        H2, dH2 = H.flip(0), [-dH[1], -dH[0]]
        parts = []
        for v, dv in ((H, dH), (H2, dH2)):
            parts.append(to_matsubara(lat.interior(v * Gm), lat.interior(v[0] * dg0 + dv[0] * Gm[0]),
                                      lat.interior(v[nw0] * dgb + dv[1] * Gm[nw0])))
        # the first frequencies read j + n, the others wrap; past the grid only the tail is left
        idx = torch.where(p1 >= 0, j + nn, torch.where(j + nn < nw0, j + nn, j + nn - nw0))
        has = (idx >= 0) & (idx < nw0)
        diff = parts[0](p1 + nn, has, idx.clamp(0, nw0 - 1)) - parts[1](p1, has | True, j)
        acc = (green(p1) * green(p1 + nn) * diff).sum(0)
        term = U * T / L2 * wt * dk * acc.imag / (4.0 * nn * PI * T)
        c3[n] = float(term.sum())
        c3k[n] = [float(term[bins == b].sum()) for b in range(nbins)]
    return {"ind_freq": None, "chijj3": c3, "chijj3_k": c3k}


def _differences(case, seed):
    """The sensitivities by central differences of the 64-bit path."""
    n, T, (tp, tpp, t3, U) = _model(case, seed)
    step = 1e-5
    rows, grad = np.zeros((3, 3)), np.zeros(3)
    for p in range(3):
        sides = []
        for sg in (1.0, -1.0):
            d = [0.0, 0.0, 0.0]
            d[p] = sg * step
            s = _Solve(case["nk0"], case["nw0"], n, T, (tp + d[2], tpp, t3, U + d[0]), mu_shift=d[1])
            sides.append(([s.Usp, s.Uch, s.D], float(_conductivity(s)["sigma"][case["nq"] - 1])))
        rows[p] = (np.array(sides[0][0]) - np.array(sides[1][0])) / (2.0 * step)
        grad[p] = (sides[0][1] - sides[1][1]) / (2.0 * step)
    return {"sum_rules": rows, "grad": grad, "dD": rows[:, 2].copy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        if case["points"] > 64:
            return None
        rows = [_Solve(int(r[0]), int(r[1]), r[2], r[3], tuple(r[4:8])).scalars() for r in _points(case, seed)]
        return {"scalars": np.array(rows), "status": None}
    if kind == "scan":
        (tp, tpp, t3, U), dens, temp = _scan(case, seed)
        dens, temp = np.linspace(*dens, case["densities"]), np.linspace(*temp, case["temperatures"])
        rows = dict.fromkeys(SCAN)
        full = [_Solve(case["nk0"], case["nw0"], n, T, (tp, tpp, t3, U), stop="roots") for n in dens for T in temp]
        rows["n"], rows["T"] = np.repeat(dens, len(temp)), np.tile(temp, len(dens))
        for col, v in (("mu0", "mu0"), ("Usp", "Usp"), ("Uch", "Uch"), ("dblOcc", "D"), ("chi0max", "chi0max")):
            rows[col] = np.array([getattr(s, v) for s in full])
        return {"rows": rows, "status": None}
    if kind == "pade":
        x, y, z = _pade(case, seed)
        g, coef = y.copy(), np.zeros_like(y)
        coef[:, 0] = g[:, 0]
        for m in range(1, x.shape[1]):
            g[:, m:] = (g[:, m - 1:m] - g[:, m:]) / ((x[:, m:] - x[:, m - 1:m]) * g[:, m:])
            coef[:, m] = g[:, m]
        v = np.zeros((x.shape[0], len(z)), dtype=complex)
        for m in range(x.shape[1] - 1, 0, -1):  # the continued fraction from its far end
            v = coef[:, m:m + 1] * (z[None, :] - x[:, m - 1:m]) / (1.0 + v)
        return coef[:, :1] / (1.0 + v)
    if kind == "gradient":
        return _differences(case, seed)
    s = _Solve(case["nk0"], case["nw0"], *_model(case, seed))
    if kind in ("solve", "driver"):
        out = {"scalars": s.scalars(), "sigma": s.sigma.cpu().numpy()}
        if kind == "driver":
            half = _Solve(case["nk0"] // 2, case["nw0"] // 2, *_model(case, seed), stop="roots")
            out["difference"] = np.array([abs((s.Usp - half.Usp) / s.Usp), abs((s.Uch - half.Uch) / s.Uch)])
        return out
    if kind == "aslamazov_larkin":
        out = _conductivity(s)
        return {**{k: out[k] for k in ("chijj1", "chijj2", "kx0")}, **_aslamazov_larkin(s, case["mmin"], case["bins"])}
    out = _conductivity(s, case["bins"])
    out["sigma"], out["bubble"] = out["sigma"][:case["nq"]], out["bubble"][:case["nq"]]
    out["scalars"] = s.scalars()
    return out
