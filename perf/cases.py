"""What is timed of this package: forwards, Jacobians, gradients and updates.

Meshes, models and surveys are the seeded synthetic ones of the benchmark
configurations (titatest_gb300.synth) at other sizes: quadrilaterals of
1 m x 0.5 m growing downwards, a draped topography, or the same grid split
into triangles; electrodes along the surface; log-normal resistivities and
phases of a random field.  exact() restates the arithmetic in 64 bits with
torch alone (element matrices, mixed boundary, block-tridiagonal elimination
by mesh columns with two refinement steps, sensitivities, the conjugate
gradient update, the covariance diagonals).
"""
import math

import numpy as np
import torch

from titatest_gb300 import MIXED, PLAIN, CRMod, formats, regularization, synth
from titatest_gb300.autograd import CRTomoMisfit
from titatest_gb300.crmod import rwaven
from titatest_gb300.ensemble import Ensemble


def _case(op, nx, nz, ne, nmeas, prec, tri=False, mode=0, count=1, ltri=0):
    return {"op": op, "nx": nx, "nz": nz, "ne": ne, "nmeas": nmeas, "prec": prec, "tri": tri, "mode": mode,
            "count": count, "ltri": ltri}


def listed():
    out = []

    def add(name, *a, **k):
        out.append(dict(_case(*a, **k), name=name))

    # a small CRMod run in the reference's arithmetic: host arrays in, voltages out (the smallest call)
    add("line_plain", "forward_host", 60, 20, 30, 180, "plain")
    # the same line in mixed precision with its Jacobian in a host array
    add("line_mixed_jacobian", "unit_host", 60, 20, 30, 180, "mixed")
    # a field profile's forward at the library's default refinement (every trial of an inversion's line search)
    add("profile_mixed", "forward", 200, 60, 96, 4000, "mixed")
    # forward + Jacobian as a replayed graph at the loose refinement setting of the benchmark
    add("profile_unit_graph", "unit_graph", 200, 60, 96, 4000, "mixed")
    # a field profile's forward in complex128
    add("profile_plain", "forward", 160, 50, 64, 2000, "plain")
    # CRTomo's Jacobian of log V on the device, both precisions
    add("jacobian_plain", "sens", 120, 40, 64, 2000, "plain", mode=1)
    add("jacobian_mixed", "sens", 200, 60, 96, 4000, "mixed", mode=1)
    # misfit and its gradient through autograd on a triangle mesh (forward, adjoint solves, contraction)
    add("gradient_triangles", "gradient", 150, 60, 64, 2000, "mixed", tri=True)
    # the preconditioned CG of one Gauss-Newton update
    add("update_cg", "update", 160, 50, 64, 2000, "plain")
    # covariance and resolution diagonals after an inversion
    add("uncertainty", "mcm", 80, 30, 40, 600, "plain", ltri=1)
    # a large survey's forward
    add("large_mixed", "forward", 300, 80, 128, 6000, "mixed")
    # a Monte-Carlo ensemble of uneven meshes
    add("ensemble_mixed", "ensemble", 160, 50, 64, 2000, "mixed", count=8)
    return out


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["forward_host", "unit_host", "forward", "forward", "unit_graph", "forward_plain", "sens", "gradient",
                     "update", "mcm", "ensemble"])
    prec = rng.choice(["plain", "mixed"])
    big = (300, 80, 128)
    if op in ("unit_host", "forward_host"):
        big = (90, 30, 40)
    elif op in ("unit_graph", "gradient", "ensemble"):
        prec, big = "mixed", (200, 60, 96)
    elif op == "forward":
        prec = "mixed"
    elif op == "forward_plain":
        op, prec, big = "forward", "plain", (160, 50, 64)
    elif op in ("update", "mcm") or (op == "sens" and prec == "plain"):
        prec, big = "plain", (90, 34, 48) if op == "mcm" else (160, 50, 64)
    elif op == "sens":
        big = (200, 60, 96)
    nx = _log_int(rng, 40, big[0])
    nz = min(_log_int(rng, 15, big[1]), nx - 5)
    ne = rng.randint(24, max(24, min(big[2], nx - 6)))
    nmeas = _log_int(rng, 200, {"mcm": 600, "update": 2000, "sens": 2000}.get(op, 4000))
    return _case(op, nx, nz, ne, nmeas, prec, tri=(op in ("forward", "gradient") and rng.random() < 0.4),
                 mode=rng.randint(0, 1) if op == "sens" else 0,
                 count=rng.randint(3, 8) if op == "ensemble" else 1, ltri=rng.randint(0, 1))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _problem(nx, nz, ne, nmeas, tri, seed):
    rng = np.random.default_rng(seed)
    step = 2 if 2 * (ne - 1) <= nx - 2 else 1
    first = (nx - step * (ne - 1)) // 2
    xs = np.arange(nx + 1, dtype=float) - first
    d, h = [0.0], 0.5
    while len(d) <= nz:  # the lower third of the rows grows by 1.1 a row
        h *= 1.1 if len(d) > 2 * nz // 3 else 1.0
        d.append(d[-1] + h)
    topo = synth._topography(xs, rng, amp=min(2.0, 0.05 * nx))
    grid, surface, _, _ = synth._quad_grid(xs, np.array(d), topo, triangles=tri, jitter=0.2 if tri else 0.0, rng=rng)
    mag, pha = synth.random_model(grid, rng)
    enodes = first + step * np.arange(ne)
    if ne <= 30:
        quads = synth.dipole_dipole(ne, [1], range(1, 9))
    else:
        quads = synth._subsample(synth.dipole_dipole(ne, range(1, 5), range(1, 9)), (nmeas + 1) // 2, rng) + \
            synth._subsample(synth.wenner_schlumberger(ne, range(1, 5), range(1, 9)), nmeas // 2, rng)
    return synth._finish("case", grid, surface, enodes, quads, mag, pha, nx, nz, triangles=tri)


def _problems(c, seed):
    """The ensemble's meshes: from a quarter of the case's width and depth up to it."""
    out = []
    for q in range(c["count"]):
        f = 0.25 + 0.75 * (q + 0.5) / c["count"]
        nx, nz = max(30, int(f * c["nx"])), max(10, int(f * c["nz"]))
        ne = min(c["ne"], nx - 6)
        out.append(_problem(nx, nz, ne, max(100, int(f * c["nmeas"])), False, seed * 1000 + q))
    return out


def _data(p, seed, nanz):
    """Noise and error model of the inversion cases: 3 % and 1 mrad on -log V."""
    rng = np.random.default_rng(seed + 7)
    noise = 0.03 * rng.standard_normal(nanz) + 1e-3j * rng.standard_normal(nanz)
    wmatd = 1.0 / (0.03 ** 2 * (1.0 + rng.uniform(0, 1, nanz)))
    return noise, wmatd


def _smoothness(p, ltri):
    if ltri == 0:
        return None, regularization.bsmatmreg(p.grid, p.nx, p.nz)
    nb = regularization.bnachbar(p.grid)
    return nb, regularization.bsmatmtri(p.grid, nb)


LAM = {"update": 5e4, "mcm": 1e3}  # as in an inversion's first iterations; near its end


def prepare(case, seed):
    c = case
    if c["op"] == "ensemble":
        return {"c": c, "ens": Ensemble(_problems(c, seed), refine_tol=1e-10)}
    p = _problem(c["nx"], c["nz"], c["ne"], c["nmeas"], c["tri"], seed)
    nanz, manz = p.survey.nanz, p.grid.elanz
    m = CRMod(p.grid, p.survey, *rwaven(p.grid, p.survey), precision=PLAIN if c["prec"] == "plain" else MIXED)
    s = {"c": c, "p": p, "m": m, "sigma": p.sigma}
    if c["op"] in ("forward", "unit_graph"):
        m.set_stream(torch.cuda.current_stream().cuda_stream)
        s["sig"] = torch.from_numpy(p.sigma).cuda()
        s["volt"] = torch.zeros(nanz, dtype=torch.complex128, device="cuda")
    if c["op"] == "unit_graph":
        m.set_refinement(8, 0.1)
    if c["op"] in ("sens", "update", "mcm"):
        out = m.forward(p.sigma, volt_mode=1)
    if c["op"] in ("sens", "unit_graph"):
        m.set_stream(torch.cuda.current_stream().cuda_stream)
        s["sens"] = torch.zeros((manz, nanz), dtype=torch.complex128, device="cuda")
    if c["op"] == "gradient":
        # data: the model's response with noise; the gradient is asked at a homogeneous start model
        v = m.forward(p.sigma)["volt"]
        noise, wmatd = _data(p, seed, nanz)
        s["phi"] = CRTomoMisfit(m, -np.log(v) + noise, wmatd).cuda()
        s["model"] = torch.full((manz,), complex(math.log(0.01), 0.015), dtype=torch.complex128, device="cuda")
    if c["op"] in ("update", "mcm"):
        m.sens_on_device(1)
        noise, s["wmatd"] = _data(p, seed, nanz)
        s["wdfak"] = np.ones(nanz, np.int32)
        s["sigmaa"], s["dat"] = out["sigmaa"], out["sigmaa"] + noise
        s["nachbar"], s["smatm"] = _smoothness(p, c["ltri"])
        s["par"] = np.log(p.sigma)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    s, c = state, state["c"]
    op = c["op"]
    if op == "ensemble":
        return [r["volt"] for r in s["ens"].run(sens_mode=None)]
    m = s["m"]
    if op == "forward_host":
        return m.forward(s["sigma"])
    if op == "unit_host":
        out = m.forward(s["sigma"])
        # the mixed Jacobian is good to 1e-5: it is kept in complex64
        return [out["volt"], m.bsens().astype(np.complex64)]
    if op == "forward":
        m.forward_device(s["sig"].data_ptr(), s["volt"].data_ptr())
        return s["volt"]
    if op == "unit_graph":
        m.forward_sens_graph(s["sig"].data_ptr(), s["volt"].data_ptr(), 0, s["sens"].data_ptr())
        # this setting stands for voltages good to 1e-6 and a Jacobian good to 1e-5: both are kept in complex64
        return [s["volt"].to(torch.complex64), s["sens"].to(torch.complex64)]
    if op == "sens":
        m.sens_device(c["mode"], s["sens"].data_ptr())
        return s["sens"] if c["prec"] == "plain" else s["sens"].to(torch.complex64)
    if op == "gradient":
        model = s["model"].clone().requires_grad_(True)
        loss = s["phi"](model)
        loss.backward()
        return [loss.detach(), model.grad]
    if op == "update":
        par, dpar, cgfac, cgres, ncg = m.update(s["wmatd"], s["wdfak"], s["dat"], s["sigmaa"], c["ltri"], s["smatm"],
                                                nx=s["p"].nx, nachbar=s["nachbar"], lam=LAM[op], par=s["par"])
        return {"par": par, "dpar": dpar, "cgfac": cgfac, "cgres": cgres, "ncg": ncg}
    assert op == "mcm"
    return m.mcm(s["wmatd"], s["wdfak"], c["ltri"], s["smatm"], nx=s["p"].nx, nachbar=s["nachbar"], lam=LAM[op])


def work(case):
    """Least work of a pass.  Forward: per wavenumber one elimination of the band matrix in its narrow order
    (4 n b^2), per wavenumber and electrode two sweeps (16 n b); sigma read, voltages written.  Jacobian: per
    element, wavenumber and electrode the product with the element matrix, per measurement the dot product;
    the potentials at the nodes read once and J written.  CG: two products with J a step (30 steps)."""
    c = case
    K = 13.0

    def forward(nx, nz, ne):
        n, b = (nx + 1.0) * (nz + 1.0), min(nx, nz) + 2.0
        return K * 4 * n * b * b + K * ne * 16 * n * b

    if c["op"] == "ensemble":
        f = [0.25 + 0.75 * (q + 0.5) / c["count"] for q in range(c["count"])]
        return {"bytes": sum(16 * (c["nx"] * c["nz"] * g * g + c["nmeas"] * g) for g in f),
                "flops": sum(forward(g * c["nx"], g * c["nz"], c["ne"]) for g in f)}
    cells, nanz = c["nx"] * c["nz"] * (2 if c["tri"] else 1), c["nmeas"]
    fw, io = forward(c["nx"], c["nz"], c["ne"]), 16.0 * (cells + nanz)
    nodes = (c["nx"] + 1.0) * (c["nz"] + 1.0)
    J = 16.0 * cells * nanz
    js = K * cells * (c["ne"] * 4 * 4 * 4 + nanz * 4 * 8.0)
    if c["op"] in ("forward_host", "forward"):
        return {"bytes": io, "flops": fw}
    if c["op"] in ("unit_host", "unit_graph"):
        return {"bytes": io + J, "flops": fw + js}
    if c["op"] == "sens":
        return {"bytes": K * c["ne"] * nodes * 16 + J, "flops": js}
    if c["op"] == "gradient":
        return {"bytes": 2 * io, "flops": fw + K * c["ne"] * 16 * nodes * (min(c["nx"], c["nz"]) + 2)}
    if c["op"] == "update":
        return {"bytes": J * 30, "flops": 30 * 16.0 * cells * nanz}
    return {"bytes": J, "flops": 2.0 * nanz * cells ** 2 + (2 / 3) * cells ** 3 + 4.0 * nanz * cells ** 2}


# ---------------------------------------------------------------------------
# the same in 64 bits, by torch alone
# ---------------------------------------------------------------------------
_TRI = [[[1, -1, 0], [-1, 1, 0], [0, 0, 0]], [[2, -1, -1], [-1, 0, 1], [-1, 1, 0]], [[1, 0, -1], [0, 0, 0], [-1, 0, 1]]]


def _triangles(x, y):
    """Stiffness and mass matrices (e, 3, 3) of linear triangles with corners x, y (e, 3)."""
    x21, x31, y21, y31 = x[:, 1] - x[:, 0], x[:, 2] - x[:, 0], y[:, 1] - y[:, 0], y[:, 2] - y[:, 0]
    det = x21 * y31 - x31 * y21
    a, b, c = (x31 ** 2 + y31 ** 2) / det, -(x31 * x21 + y31 * y21) / det, (x21 ** 2 + y21 ** 2) / det
    t = torch.tensor(_TRI, dtype=torch.float64, device=x.device)
    S = (a[:, None, None] * t[0] + b[:, None, None] * t[1] + c[:, None, None] * t[2]) / 2
    M = det[:, None, None] / 24 * (1 + torch.eye(3, dtype=torch.float64, device=x.device))
    return S, M


def _poly(t, coef):
    v = torch.zeros_like(t)
    for c in reversed(coef):
        v = v * t + c
    return v


def _k0k1(x):
    """K0, K1 by the polynomials of Abramowitz & Stegun 9.8.1, 9.8.3, 9.8.5-9.8.8 (0 beyond 500)."""
    t = (x / 3.75) ** 2
    i0 = _poly(t, [1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813])
    i1 = x * _poly(t, [0.5, 0.87890594, 0.51498869, 0.15084934, 0.02658733, 0.00301532, 0.00032411])
    q = x * x / 4
    l = torch.log(x / 2)
    a0 = -l * i0 + _poly(q, [-0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698, 0.00010750, 0.0000074])
    a1 = l * i1 + _poly(q, [1.0, 0.15443144, -0.67278579, -0.18156897, -0.01919402, -0.00110404, -0.00004686]) / x
    u, f = 2 / x, torch.exp(-x) / torch.sqrt(x)
    b0 = f * _poly(u, [1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872, -0.00251540, 0.00053208])
    b1 = f * _poly(u, [1.25331414, 0.23498619, -0.03655620, 0.01504268, -0.00780353, 0.00325614, -0.00068245])
    far = x > 500
    return torch.where(x <= 2, a0, b0).masked_fill(far, 0.0), torch.where(x <= 2, a1, b1).masked_fill(far, 0.0)


class _Exact:
    """A problem's matrices on the device, nodes in mesh columns (column-major: node = column * h + row)."""

    def __init__(self, p):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.p, self.dev, g = p, dev, p.grid
        self.h, self.w = p.nz + 1, p.nx + 1
        nat = np.asarray(g.snr, np.int64) - 1  # band position -> node of the generator, row by row
        pos = (nat % self.w) * self.h + nat // self.w

        def up(a, **k):
            return torch.as_tensor(np.ascontiguousarray(a), device=dev, **k)

        xy = np.zeros((2, g.sanz))
        xy[:, pos] = np.stack(g.node_xy())
        self.x, self.y = up(xy[0]), up(xy[1])
        E, nk = g.elanz, int(g.selanz[0])
        self.E, self.nk = E, nk
        self.conn = up(pos[g.nrel[:E, :nk].astype(np.int64) - 1])
        x, y = self.x[self.conn], self.y[self.conn]
        if nk == 3:
            self.S, self.M = _triangles(x, y)
        else:  # four triangles about the diagonals' intersection, the centre condensed
            a1 = (y[:, 2] - y[:, 0]) / (x[:, 2] - x[:, 0])
            dx2 = x[:, 3] - x[:, 1]
            a2 = (y[:, 3] - y[:, 1]) / dx2
            xc = (a1 * x[:, 0] - y[:, 0] - a2 * x[:, 1] + y[:, 1]) / (a1 - a2)
            yc = y[:, 0] + a1 * (xc - x[:, 0])
            x5, y5 = torch.cat([x, xc[:, None]], 1), torch.cat([y, yc[:, None]], 1)
            self.S = torch.zeros((E, 5, 5), dtype=torch.float64, device=dev)
            self.M = torch.zeros_like(self.S)
            for t in ([0, 1, 4], [1, 2, 4], [4, 2, 3], [0, 4, 3]):
                s, m = _triangles(x5[:, t], y5[:, t])
                for i in range(3):
                    for j in range(3):
                        self.S[:, t[i], t[j]] += s[:, i, j]
                        self.M[:, t[i], t[j]] += m[:, i, j]
        kw, wi = rwaven(g, p.survey)
        self.kw, self.wi = up(kw), up(wi) / math.pi
        nm = int(g.nelanz[2])  # mixed boundary lines, listed last
        self.bn = up(pos[g.nrel[-nm:, :2].astype(np.int64) - 1])
        self.be = up(np.asarray(g.rnr[-nm:], np.int64) - 1)
        self.en = up(pos[np.asarray(p.survey.enr, np.int64) - 1])
        st, vn = np.asarray(p.survey.strnr, np.int64), np.asarray(p.survey.vnr, np.int64)
        self.el = [up(a - 1) for a in (st % 10000, st // 10000, vn % 10000, vn // 10000)]  # all four present
        self.strom = up(np.asarray(p.survey.strom, float))

    def element(self, k):
        """(e, nk, nk) element matrices at wavenumber k."""
        m = self.S + self.kw[k] ** 2 * self.M
        return m if self.nk == 3 else m[:, :4, :4] - m[:, :4, 4:] * m[:, 4:, :4] / m[:, 4:, 4:]

    def boundary(self, k):
        """(l, line, 2, 2) boundary matrices over sigma at wavenumber k."""
        x, y, k_ = self.x[self.bn], self.y[self.bn], self.kw[k]
        xs, ys = self.x[self.en][:, None], self.y[self.en][:, None]
        dx, dy = x[:, 1] - x[:, 0], y[:, 1] - y[:, 0]
        ln = torch.sqrt(dx * dx + dy * dy)
        ex, ym, yp = x.mean(1) - xs, y.mean(1) - ys, y.mean(1) + ys
        rm, rp = torch.sqrt(ex * ex + ym * ym), torch.sqrt(ex * ex + yp * yp)
        cm, cp = (-ex * dy + ym * dx) / rm / ln, (-ex * dy + yp * dx) / rp / ln
        (k0m, k1m), (k0p, k1p) = _k0k1(rm * k_), _k0k1(rp * k_)
        den = k0m + k0p
        b = torch.where(den == 0, (cm + cp) / 2, (cm * k1m + cp * k1p) / torch.where(den == 0, torch.ones_like(den), den))
        mass = torch.tensor([[2.0, 1.0], [1.0, 2.0]], dtype=torch.float64, device=self.dev) / 6
        return (k_ * b * ln)[:, :, None, None] * mass

    def solver(self, sigma, k):
        """(solve, apply) of the systems of wavenumber k, one per electrode: arrays (l, n)."""
        h, w, L, n = self.h, self.w, len(self.en), self.h * self.w
        Ke, Kb = self.element(k) * sigma[:, None, None], self.boundary(k) * sigma[self.be][:, None, None]

        def apply(v):
            r = torch.zeros_like(v)
            r.index_add_(1, self.conn.reshape(-1), torch.einsum("eij,lej->lei", Ke, v[:, self.conn]).reshape(L, -1))
            r.index_add_(1, self.bn.reshape(-1), torch.einsum("lbij,lbj->lbi", Kb, v[:, self.bn]).reshape(L, -1))
            return r

        D = torch.zeros((w * h * h,), dtype=torch.complex128, device=self.dev)
        U = torch.zeros_like(D)  # U[j]: rows of column j, columns of column j + 1
        i, j = self.conn[:, :, None].expand_as(Ke).reshape(-1), self.conn[:, None, :].expand_as(Ke).reshape(-1)
        v, ci, cj = Ke.reshape(-1), i // h, j // h
        at = (ci * h + i % h) * h + j % h
        D.index_add_(0, at[ci == cj], v[ci == cj])
        U.index_add_(0, at[cj == ci + 1], v[cj == ci + 1])
        D, U = D.reshape(w, h, h), U.reshape(w, h, h)
        i, j = self.bn[:, :, None].expand(-1, 2, 2).reshape(-1), self.bn[:, None, :].expand(-1, 2, 2).reshape(-1)
        vb, ci, cj = Kb.reshape(L, -1), i // h, j // h
        at = (i % h) * h + j % h
        P, Uc = [], []
        for c in range(w):
            S = D[c].repeat(L, 1, 1).reshape(L, -1)
            q = (ci == c) & (cj == c)
            S.index_add_(1, at[q], vb[:, q])
            Uj = U[c].repeat(L, 1, 1).reshape(L, -1)
            q = (ci == c) & (cj == c + 1)
            Uj.index_add_(1, at[q], vb[:, q])
            S = S.reshape(L, h, h)
            if c:
                S = S - Uc[-1].transpose(1, 2) @ (P[-1] @ Uc[-1])
            P.append(torch.linalg.inv(S))
            Uc.append(Uj.reshape(L, h, h))

        def once(b):
            y = [b[:, c * h:(c + 1) * h, None] for c in range(w)]
            for c in range(1, w):
                y[c] = y[c] - Uc[c - 1].transpose(1, 2) @ (P[c - 1] @ y[c - 1])
            for c in range(w - 1, -1, -1):
                y[c] = P[c] @ (y[c] - Uc[c] @ y[c + 1] if c < w - 1 else y[c])
            return torch.cat(y, 1)[:, :, 0]

        def solve(b):
            x = once(b)
            for _ in range(2):
                x = x + once(b - apply(x))
            return x

        return solve, apply, Kb

    def measure(self, hp):
        """Voltages from hp (l, n): potentials of electrode l at every node."""
        e1, e2, e3, e4 = self.el
        at = hp[:, self.en]
        return (at[e2, e4] - at[e1, e4]) - (at[e2, e3] - at[e1, e3])

    def forward(self, sigma, keep=True):
        L, n = len(self.en), self.h * self.w
        src = torch.zeros((L, n), dtype=torch.complex128, device=self.dev)
        src[torch.arange(L, device=self.dev), self.en] = 1.0
        self.kpot, hp = [], 0
        for k in range(len(self.kw)):
            x = self.solver(sigma, k)[0](src)
            hp = hp + x * self.wi[k]
            if keep:
                self.kpot.append(x)
        self.volt = self.measure(hp)
        return self.volt

    def sens(self, sigma, mode):
        """(element, measurement) sensitivities."""
        e1, e2, e3, e4 = self.el
        J = torch.zeros((self.E, len(e1)), dtype=torch.complex128, device=self.dev)
        step = max(1, int(4e8 / (16 * self.nk * len(e1))))
        for k in range(len(self.kw)):
            Ke, U = self.element(k) * self.wi[k], self.kpot[k]
            for a in range(0, self.E, step):
                u = U[:, self.conn[a:a + step]].permute(1, 2, 0)  # (element, node, electrode)
                du, dv = u[:, :, e2] - u[:, :, e1], u[:, :, e4] - u[:, :, e3]
                J[a:a + step] += (dv * (Ke[a:a + step].to(torch.complex128) @ du)).sum(1)
        return -J * self.strom if mode == 0 else J * sigma[:, None] / self.volt

    def gradient(self, sigma, g):
        """sum_i g_i dV_i/dsigma by adjoint solves."""
        e1, e2, e3, e4 = self.el
        L, n = len(self.en), self.h * self.w
        src = torch.zeros((L * n,), dtype=torch.complex128, device=self.dev)
        for a, b, sgn in ((e2, e4, 1), (e2, e3, -1), (e1, e4, -1), (e1, e3, 1)):
            src.index_add_(0, a * n + self.en[b], sgn * g)
        src = src.reshape(L, n)
        out = torch.zeros((self.E,), dtype=torch.complex128, device=self.dev)
        for k in range(len(self.kw)):
            solve, _, _ = self.solver(sigma, k)
            lam, x = solve(src), self.kpot[k]
            Ke = self.element(k).to(torch.complex128)
            out -= self.wi[k] * torch.einsum("lei,eij,lej->e", lam[:, self.conn], Ke, x[:, self.conn])
            Kb = self.boundary(k).to(torch.complex128)
            t = torch.einsum("lbi,lbij,lbj->b", lam[:, self.bn], Kb, x[:, self.bn])
            out.index_add_(0, self.be, -self.wi[k] * t)
        return out


def _too_long(c):
    n, b, K = (c["nx"] + 1.0) * (c["nz"] + 1.0), c["nz"] + 1.0, 14
    return n * b * b * K * c["ne"] * 90 > 6e12  # about 11 b^3 complex steps a column, at an FP64 TFLOP/s


def _smooth(c, p, sm, nb, v):
    """The smoothness operator on v (manz)."""
    r = sm[0 if c["ltri"] == 0 else -1] * v
    if c["ltri"] == 0:
        nx = p.nx
        r[1:] += sm[1, :-1] * v[:-1]
        r[:-1] += sm[1, :-1] * v[1:]
        r[nx:] += sm[2, :-nx] * v[:-nx]
        r[:-nx] += sm[2, :-nx] * v[nx:]
        return r
    for q in range(nb.shape[0] - 1):
        has = nb[q] > 0
        r[has] += sm[q][has] * v[nb[q][has].long() - 1]
    return r


def exact(case, seed):
    c = case
    if c["op"] == "ensemble":
        ps = _problems(c, seed)
        return [_Exact(p).forward(torch.as_tensor(p.sigma).to(_Exact(p).dev), False).cpu().numpy() for p in ps]
    if _too_long(c):
        return None
    p = _problem(c["nx"], c["nz"], c["ne"], c["nmeas"], c["tri"], seed)
    x = _Exact(p)
    sigma = torch.as_tensor(p.sigma).to(x.dev)
    nanz = p.survey.nanz
    V = x.forward(sigma, c["op"] not in ("forward", "forward_host"))
    if c["op"] == "forward_host":
        return {"volt": V, "sigmaa": V}
    if c["op"] == "forward":
        return V
    if c["op"] == "unit_host":
        return [V, x.sens(sigma, 0).T]
    if c["op"] == "unit_graph":
        return [V, x.sens(sigma, 0)]
    if c["op"] == "sens":
        return x.sens(sigma, c["mode"])
    noise, wmatd = (torch.as_tensor(a).to(x.dev) for a in _data(p, seed, nanz))
    if c["op"] == "gradient":
        dobs = -torch.log(V) + noise
        s0 = torch.exp(torch.full((x.E,), complex(math.log(0.01), 0.015), dtype=torch.complex128, device=x.dev))
        V = x.forward(s0)
        r = -torch.log(V) - dobs
        g = x.gradient(s0, wmatd * r.conj() * (-1 / V))
        return [(wmatd * r.abs() ** 2).sum(), 2 * (g * s0).conj()]
    J = x.sens(sigma, 1).T.contiguous()  # (measurement, element)
    nb, sm = _smoothness(p, c["ltri"])
    lam = LAM[c["op"]]
    if c["op"] == "mcm":
        Js = torch.sqrt(wmatd)[:, None] * J
        ata = Js.real.T @ Js.real + Js.imag.T @ Js.imag
        reg = ata.clone()
        i = torch.arange(x.E, device=x.dev)
        s = torch.as_tensor(sm).to(x.dev)
        reg[i, i] += lam * s[0 if c["ltri"] == 0 else -1]
        if c["ltri"] == 0:
            for d, row in ((1, 1), (p.nx, 2)):
                reg[i[:-d], i[d:]] += lam * s[row, :-d]
                reg[i[d:], i[:-d]] += lam * s[row, :-d]
        else:  # as many leading slots as a cell has neighbours, both triangles
            for q in range(nb.shape[0] - 1):
                has = np.flatnonzero((nb[q] > 0) & (nb[-1] > q))
                a, b = torch.as_tensor(has).to(x.dev), torch.as_tensor(nb[q][has].astype(np.int64) - 1).to(x.dev)
                v = ata[a, b] + lam * s[q][a]
                reg[a, b] = v
                reg[b, a] = v
        cov = torch.linalg.inv(reg)
        res = cov @ ata
        return {"ata": ata.diagonal(), "reg": reg.diagonal(), "cov1": cov.diagonal(), "res": res.diagonal(),
                "cov2": (res * cov).sum(1)}
    # the update: preconditioned conjugate gradients on J^H W J + lam R
    s, nbt = torch.as_tensor(sm).to(x.dev), None if nb is None else torch.as_tensor(nb).to(x.dev)
    par = torch.log(sigma)
    f = 1 / torch.sqrt((J.abs() ** 2 * wmatd[:, None]).sum(0) + lam * s[0 if c["ltri"] == 0 else -1])
    r = (J.conj().T @ (wmatd * noise) - lam * _smooth(c, p, s, nbt, par)) * f
    d, q, dr1, res = torch.zeros_like(r), torch.zeros_like(r), 1.0, np.zeros(102)
    for k in range(1, 101):
        dr = float((r.abs() ** 2).sum())
        if k == 1:
            dr0, beta = dr * 1e-4, 0.0
        elif dr <= dr0:
            k -= 1
            break
        else:
            beta = dr / dr1
        q = r + beta * q
        t = (J.conj().T @ (wmatd * (J @ (f * q))) + lam * _smooth(c, p, s, nbt, f * q)) * f
        alpha = dr / float((q.conj() * t).sum().real)
        d, r, dr1 = d + alpha * q, r - alpha * t, dr
        res[k] = 1e-4 * dr / dr0
    res[0] = k
    return {"par": par + f * d, "dpar": f * d, "cgfac": f, "cgres": res, "ncg": None}
