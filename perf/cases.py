"""The calls a user of the framework makes, at the sizes they make them, for timing and for comparing results.

``listed()`` holds one case per kind of work; ``draw(rng)`` gives further cases of the same
ranges.  ``prepare`` builds what a program has in hand before the call (links, sources,
operator and solver objects), ``run`` is one pass through the public entry points, ``exact``
the same result in 64-bit torch without this package, ``work`` the bytes and operations the
result cannot do without.

Links are SU(N) matrices near the identity, as rough as the thermalised ones the solvers
meet; fermions are antiperiodic in time; sources are unit complex Gaussian.
"""
import math

import numpy as np
import torch

from tfleonardym_b200 import (approximations, boundary_conditions, dirac, dirac_solver, fermion_action,
                              fermion_measurements, gauge_action, hmc, measurements, smearing)
from tfleonardym_b200 import lattice as lt

dirac_solver.VERBOSE = False

C128 = torch.complex128


def listed():
    return [
        # the smallest call: one 2D SU(2) source in FP64 (HMC on two-dimensional lattices); latency
        dict(name="solve_2d_f64", kind="solve", geometry="24x16", nc=2, kappa=0.13, nrhs=1, precision="f64",
             tol=1e-10, delta=0.1, hermitian=True),
        # one 4D source at a time in FP64: a single propagator column, an HMC energy
        dict(name="solve_4d_f64", kind="solve", geometry="16x16x16x16", nc=3, kappa=0.13, nrhs=1, precision="f64",
             tol=1e-10, delta=0.1, hermitian=False),
        # the served workload: 16 sources per call, FP16 inner iterations
        dict(name="solve_4d_f16_16rhs", kind="solve", geometry="16x16x16x16", nc=3, kappa=0.13, nrhs=16,
             precision="f16", tol=1e-10, delta=0.01, hermitian=False),
        # a production lattice, several sources, FP32 inner iterations
        dict(name="solve_24c48_f32", kind="solve", geometry="24x24x24x48", nc=3, kappa=0.13, nrhs=4,
             precision="f32", tol=1e-10, delta=0.1, hermitian=False),
        # many small independent lattices in one call (ensembles, parameter scans)
        dict(name="lattices_3d_f32", kind="lattices",
             geometry="8x8x8,16x10x12,14x8x10,16x16x16,10x12x8,12x12x14,8x16x10,14x14x8", nc=2, kappa=0.12, nrhs=4,
             precision="f32", tol=1e-10, hermitian=False),
        # one RHMC force: multishift solve over the poles, operator on all of them, fused force
        dict(name="rhmc_force", kind="rhmc_force", geometry="12x12x12x24", nc=3, kappa=0.125, poles=8,
             precision="f64", tol=1e-11),
        # the operator itself in the reference layout: the inner call of a user's own Krylov solver
        dict(name="apply_32", kind="apply", representation="fundamental", geometry="32x32x32x32", nc=3, kappa=0.13,
             nvec=1, hermitian=True),
        # the operator on a stack of vectors (poles, propagator columns)
        dict(name="apply_batch", kind="apply", representation="fundamental", geometry="16x16x16x32", nc=3,
             kappa=0.13, nvec=12, hermitian=False),
        # adjoint fermions (supersymmetric Yang-Mills): the operator
        dict(name="apply_adjoint", kind="apply", representation="adjoint", geometry="16x16x16x16", nc=3, kappa=0.12,
             nvec=1, hermitian=True),
        # adjoint fermions: the force of a rational approximation's poles
        dict(name="force_adjoint", kind="force", representation="adjoint", geometry="8x8x8x16", nc=3, kappa=0.12,
             poles=4),
        # pure-gauge molecular dynamics: force kicks and link drifts
        dict(name="md_gauge", kind="md", geometry="16x16x16x32", nc=3, beta=5.8, steps=2),
        # measurements on a stored configuration: smearing, glueball and Polyakov operators, plaquette
        dict(name="measure", kind="measure", geometry="24x24x24x48", nc=3, rho=0.4),
    ]


def _even(rng, lo, hi):
    """An even extent, log-uniform in [lo, hi]."""
    return 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, sizes log-uniform over its range (odd ones wherever the call takes
    them: the even-odd solvers need even extents)."""
    kind = rng.choice(["solve", "solve", "lattices", "rhmc_force", "apply", "apply", "force", "md", "measure",
                       "propagator"])
    kappa = round(rng.uniform(0.10, 0.135), 4)
    nc = rng.choice([2, 3])
    if kind in ("solve", "propagator"):
        nd = rng.choice([2, 3, 4, 4])
        hi = {2: (256, 256), 3: (48, 48, 48), 4: (16, 16, 16, 32)}[nd]
        geometry = [_even(rng, 6, h) for h in hi]
        case = dict(kind=kind, geometry="x".join(map(str, geometry)), nc=nc, kappa=kappa)
        if kind == "propagator":
            return dict(case, tol=1e-12, direction=rng.randrange(nd))
        return dict(case, nrhs=rng.choice([1, 1, 2, 3, 4, 7, 8, 12, 16]),
                    precision=rng.choice(["f64", "f32", "f16", "bf16"]),
                    tol=10 ** rng.uniform(-12, -10.5), delta=rng.choice([0.1, 0.03, 0.01]),
                    hermitian=nd != 3 and rng.random() < 0.5)
    if kind == "lattices":
        nd = rng.choice([2, 3, 4])
        lo, hi = {2: (8, 64), 3: (8, 16), 4: (6, 10)}[nd]
        geometry = ",".join("x".join(str(_even(rng, lo, hi)) for _ in range(nd)) for _ in range(rng.randint(2, 10)))
        return dict(kind=kind, geometry=geometry, nc=nc, kappa=kappa, nrhs=rng.randint(1, 6),
                    precision=rng.choice(["f64", "f32", "f16"]), tol=1e-11, hermitian=False)
    if kind == "rhmc_force":
        nd = rng.choice([2, 4])
        hi = {2: (96, 96), 4: (12, 12, 12, 24)}[nd]
        return dict(kind=kind, geometry="x".join(str(_even(rng, 6, h)) for h in hi), nc=nc, kappa=min(kappa, 0.125),
                    poles=rng.randint(2, 12), precision=rng.choice(["f64", "f64", "f32"]), tol=1e-11)
    if kind in ("apply", "force"):
        representation = rng.choice(["fundamental", "fundamental", "adjoint"])
        adjoint = representation == "adjoint"
        nd = rng.choice([2, 4] if adjoint or kind == "force" else [2, 3, 4])
        hi = {2: 512, 3: 64, 4: 16 if adjoint or kind == "force" else 24}[nd]
        if adjoint and kind == "force":
            hi = min(hi, 256) if nd == 2 else 10
        geometry = "x".join(str(_extent(rng, 4, hi)) for _ in range(nd))
        case = dict(kind=kind, representation=representation, geometry=geometry, nc=nc, kappa=kappa)
        if kind == "force":
            return dict(case, poles=rng.randint(1, 4 if adjoint else 10))
        return dict(case, nvec=rng.choice([1, 1, 2, 3, 8, 13]) if not adjoint else rng.choice([1, 2, 5]),
                    hermitian=nd != 3 and rng.random() < 0.5)
    if kind == "md":
        nd = rng.choice([2, 3, 4, 4])
        hi = {2: 512, 3: 64, 4: 20}[nd]
        return dict(kind=kind, geometry="x".join(str(_extent(rng, 4, hi)) for _ in range(nd)), nc=nc,
                    beta=round(rng.uniform(2.0, 6.0), 3), steps=rng.randint(1, 2))
    return dict(kind="measure", geometry="x".join(str(_extent(rng, 4, 28)) for _ in range(4)), nc=nc,
                rho=round(rng.uniform(0.2, 0.6), 3))


# ---------------------------------------------------------------------------
# inputs, made from the seed alone
# ---------------------------------------------------------------------------
def _geometries(case):
    return [tuple(int(n) for n in g.split("x")) for g in case["geometry"].split(",")]


def _ns(nd):
    return 4 if nd == 4 else 2


def _normal(gen, shape):
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=gen, dtype=torch.float64, device="cuda"))


def _generator(seed, k=0):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * int(seed) + k)
    return gen


def _links(gen, nd, nc, vol, width=0.25):
    """SU(N) links (nd, N, N, V): Gram-Schmidt of 1 + width * (complex Gaussian)."""
    m = _normal(gen, (nd, nc, nc, vol)) * width
    for i in range(nc):
        m[:, i, i] += 1
    r0 = m[:, 0] / torch.linalg.vector_norm(m[:, 0], dim=1, keepdim=True)
    if nc == 2:
        return torch.stack([r0, torch.stack([-r0[:, 1].conj(), r0[:, 0].conj()], 1)], 1).contiguous()
    r1 = m[:, 1] - (r0.conj() * m[:, 1]).sum(1, keepdim=True) * r0
    r1 = r1 / torch.linalg.vector_norm(r1, dim=1, keepdim=True)
    r2 = torch.stack([r0[:, (k + 1) % 3] * r1[:, (k + 2) % 3] - r0[:, (k + 2) % 3] * r1[:, (k + 1) % 3]
                      for k in range(3)], 1).conj()
    return torch.stack([r0, r1, r2], 1).resolve_conj().contiguous()


def _momenta(gen, nd, nc, vol):
    """Traceless anti-Hermitian Gaussian matrices (nd, N, N, V)."""
    a = _normal(gen, (nd, nc, nc, vol)) * 0.5
    p = a - a.conj().transpose(1, 2)
    tr = sum(p[:, i, i] for i in range(nc)) / nc
    for i in range(nc):
        p[:, i, i] -= tr
    return p.resolve_conj().contiguous()


def _poles(case):
    """alphas, betas of the x^(-1/2) approximation with the case's number of poles."""
    a, b, _ = approximations.zolotarev_inverse_sqrt(int(case["poles"]), 1e-2, grid=2001)
    return [float(x) for x in a], [float(x) for x in b]


def _sources(gen, case, nd, nc, vol):
    kind = case["kind"]
    if kind in ("solve", "lattices"):
        return _normal(gen, (case["nrhs"], _ns(nd), nc, vol))
    if kind == "propagator":
        return _normal(gen, (_ns(nd) * nc, _ns(nd), nc, vol))
    if kind == "rhmc_force":
        return _normal(gen, (_ns(nd), nc, vol))
    return None


def _algebra_spinor(gen, n, nd, nc, vol):
    """Adjoint spinors (n, ns, N, N, V): traceless matrices."""
    v = _normal(gen, (n, _ns(nd), nc, nc, vol))
    tr = sum(v[:, :, i, i] for i in range(nc)) / nc
    for i in range(nc):
        v[:, :, i, i] -= tr
    return v


# ---------------------------------------------------------------------------
# the program's objects, and one pass
# ---------------------------------------------------------------------------
def _operator(links, geometry, case, hermitian):
    cfg = lt.Configuration(links, geometry, int(case["nc"]), len(geometry))
    provider = boundary_conditions.time_antiperiodic_provider(-1)
    return dirac.DiracWilsonOperator(cfg, case["kappa"], hermitian,
                                     representation=case.get("representation", "fundamental"),
                                     boundary_condition_provider=provider)


def _inputs(case, seed):
    """Per lattice of the case: (geometry, links, what else the kind takes)."""
    out = []
    nc = int(case["nc"])
    for k, geometry in enumerate(_geometries(case)):
        nd, vol = len(geometry), int(np.prod(geometry))
        gen = _generator(seed, k)
        links = _links(gen, nd, nc, vol)
        kind = case["kind"]
        if kind == "apply":
            if case["representation"] == "adjoint":
                extra = _algebra_spinor(gen, case["nvec"], nd, nc, vol)
            else:
                extra = _normal(gen, (case["nvec"], _ns(nd), nc, vol))
        elif kind == "force":
            if case["representation"] == "adjoint":
                extra = [_algebra_spinor(gen, case["poles"], nd, nc, vol) for _ in range(2)]
            else:
                extra = [_normal(gen, (case["poles"], _ns(nd), nc, vol)) for _ in range(2)]
        elif kind == "md":
            extra = _momenta(gen, nd, nc, vol)
        else:
            extra = _sources(gen, case, nd, nc, vol)
        out.append((geometry, links, extra))
    return out


def prepare(case, seed):
    kind = case["kind"]
    inputs = _inputs(case, seed)
    geometry, links, extra = inputs[0]
    state = dict(kind=kind, extra=extra)
    if kind == "solve":
        state["op"] = _operator(links, geometry, case, case["hermitian"])
        state["solver"] = dirac_solver.conjugate_gradient(tol=case["tol"], precision=case["precision"],
                                                          delta=case["delta"])
    elif kind == "lattices":
        state["ops"] = [_operator(u, g, case, False) for g, u, _ in inputs]
        state["sources"] = [b for _, _, b in inputs]
        state["case"] = case
    elif kind == "propagator":
        state["op"] = _operator(links, geometry, case, False)
        state["propagator"] = dirac.Propagator(state["op"], dirac_solver.conjugate_gradient(tol=case["tol"]))
        state["direction"] = case["direction"]
    elif kind == "rhmc_force":
        q = _operator(links, geometry, case, True)
        solver = dirac_solver.multishift_cg(20000, case["tol"], precision=case["precision"])
        alphas, betas = _poles(case)
        ra = dirac.RationalApproximation(dirac.SquareOperator(q), alphas, betas, 0.0, solver)
        nf = fermion_action.n_flavor([ra], [ra], [ra], solver, q)
        nf.pseudofermions = [extra]
        state["action"] = nf
    elif kind == "apply":
        state["op"] = _operator(links, geometry, case, case["hermitian"])
    elif kind == "force":
        state["op"] = _operator(links, geometry, case, True)
        state["alphas"] = _poles(case)[0]
    else:
        state["cfg"] = lt.Configuration(links, geometry, int(case["nc"]), len(geometry))
        if kind == "md":
            state["action"] = gauge_action.yang_mills(state["cfg"], case["beta"])
            state["steps"] = [int(case["steps"])]
        else:
            state["rho"] = case["rho"]
    return state


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return state["solver"].solve(state["op"], state["extra"])
    if kind == "lattices":
        c = state["case"]
        return dirac_solver.solve_lattices(state["ops"], state["sources"], tol=c["tol"], precision=c["precision"])[0]
    if kind == "propagator":
        s = state["propagator"].apply(state["extra"])
        return s, fermion_measurements.slice_sums(s, state["op"], state["direction"])
    if kind == "rhmc_force":
        return state["action"].force()
    if kind == "apply":
        return state["op"].apply(state["extra"])
    if kind == "force":
        op = state["op"]
        force = torch.zeros_like(op.cfg.gauge_field)
        return op.accumulate_force(force, state["alphas"], state["extra"][0], state["extra"][1], symmetric=True)
    if kind == "md":
        cfg, p = hmc.integrate_om(state["cfg"], state["extra"], [state["action"]], state["steps"], 0.1)
        return cfg.gauge_field, p
    cfg = state["cfg"]
    smeared = smearing.ape_smearing(cfg, state["rho"])
    values = measurements.glueball_operators(smeared) + measurements.polyakov_operators(cfg)
    values.append(measurements.plaquette(cfg))
    return smeared.gauge_field, [np.asarray(m.value) for m in values]


# ---------------------------------------------------------------------------
# what one pass cannot do without
# ---------------------------------------------------------------------------
def _hop_flops(nd, nc):
    """Flops of all hops at one site: per direction and sign, ns/2 projected colour vectors, their
    matrix products and the accumulation."""
    ns = _ns(nd)
    return 2 * nd * (ns // 2) * (2 * nc + nc * (8 * nc - 2)) + (2 * nd - 1) * ns * nc * 2


def work(case):
    kind, nc = case["kind"], int(case["nc"])
    nbytes = flops = 0.0
    for geometry in _geometries(case):
        nd, vol = len(geometry), int(np.prod(geometry))
        ns = _ns(nd)
        links = 16.0 * nd * nc * nc * vol
        vec = 16.0 * ns * nc * vol
        adj = 16.0 * ns * nc * nc * vol
        mm = 8.0 * nc ** 3 - 2 * nc * nc  # one N x N complex product
        dslash = _hop_flops(nd, nc) * vol
        staples = nd * (nd - 1) * 2 * (2 * mm + 2 * nc * nc) * vol
        # iterations to the tolerance at these kappas (about 4 per decade on M^dag M, two M each)
        its = 8.0 * -math.log10(case.get("tol", 1e-10))
        if kind in ("solve", "lattices", "propagator"):
            n = ns * nc if kind == "propagator" else case["nrhs"]
            nbytes += links + 2 * n * vec
            flops += n * its * (2 * dslash + 8 * ns * nc * vol)
        elif kind == "rhmc_force":
            nbytes += links + vec + links
            flops += its * (2 * dslash + case["poles"] * 8 * ns * nc * vol)
        elif kind == "apply" and case["representation"] == "fundamental":
            nbytes += links + 2 * case["nvec"] * vec
            flops += case["nvec"] * dslash
        elif kind == "apply":
            nbytes += links + 2 * case["nvec"] * adj
            flops += case["nvec"] * 2 * nd * (ns // 2) * (2 * mm + 4 * nc * nc) * vol
        elif kind == "force":
            v = adj if case["representation"] == "adjoint" else vec
            nbytes += 2 * links + 2 * case["poles"] * v
            # per link and pole: U Y (and its partner), then the outer products over spin
            per = 2 * ns * (nc if case["representation"] == "adjoint" else 1) * (2 * 8.0 * nc * nc)
            flops += case["poles"] * nd * 2 * per * vol
        elif kind == "md":
            kicks = 2 * case["steps"] + 1
            nbytes += 4 * links
            flops += kicks * staples + 2 * case["steps"] * nd * 4 * mm * vol
        else:
            nbytes += 2 * links
            flops += staples + nd * 10 * mm * vol + (3 * (3 + 7) + geometry[-1]) * mm * vol
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64-bit torch
# ---------------------------------------------------------------------------
def _shift(f, geometry, mu, step=1):
    """f(x + step * mu) along the site axis."""
    nd = len(geometry)
    return torch.roll(f.reshape(f.shape[:-1] + geometry), -step, dims=mu - nd).reshape(f.shape)


def _mm(a, b):
    return torch.stack([torch.stack([sum(a[..., i, k, :] * b[..., k, j, :] for k in range(b.shape[-3]))
                                     for j in range(b.shape[-2])], -2) for i in range(a.shape[-3])], -3)


def _dag(a):
    return a.transpose(-3, -2).conj()


def _gammas(nd):
    if nd == 4:
        g = np.zeros((4, 4, 4), dtype=complex)
        for mu, (col, ph) in enumerate((((3, 2), (-1j, -1j)), ((3, 2), (-1, 1)), ((2, 3), (-1j, 1j)), ((2, 3), (1, 1)))):
            for a in range(2):
                g[mu, a, col[a]] = ph[a]
                g[mu, col[a], a] = np.conj(ph[a])
        return g
    s = np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]], dtype=complex)
    return s[:nd]


def _spin(m, v, axis):
    """Spin matrix m on the spin axis of v."""
    out = []
    for i in range(m.shape[0]):
        t = None
        for j in range(m.shape[1]):
            if m[i, j] != 0:
                w = complex(m[i, j]) * v.select(axis, j)
                t = w if t is None else t + w
        out.append(torch.zeros_like(v.select(axis, 0)) if t is None else t)
    return torch.stack(out, axis)


def _bc(links, geometry):
    u = links.clone()
    u[-1][..., geometry[-1] - 1::geometry[-1]] *= -1
    return u


class _Wilson:
    """D (or gamma_d D) on stacks (n, ns, N, V), or matrix-valued (n, ns, N, N, V) with adjoint=True."""

    def __init__(self, links, geometry, kappa, hermitian, adjoint=False):
        self.geometry, self.kappa, self.hermitian, self.adjoint = geometry, kappa, hermitian, adjoint
        self.u, self.right = _bc(links, geometry), links
        self.g = _gammas(len(geometry))

    def _act(self, u, r, v):
        """u v, and (adjoint) u v r^dag."""
        if self.adjoint:
            return _mm(_mm(u[None, None], v), _dag(r)[None, None])
        return torch.stack([sum(u[i, j] * v[:, :, j] for j in range(u.shape[1])) for i in range(u.shape[0])], 2)

    def apply(self, v):
        acc = torch.zeros_like(v)
        one = np.eye(self.g.shape[1])
        for mu in range(len(self.geometry)):
            u, r = self.u[mu], self.right[mu]
            acc += self._act(u, r, _shift(_spin(one - self.g[mu], v, 1), self.geometry, mu))
            acc += _shift(self._act(_dag(u), _dag(r), _spin(one + self.g[mu], v, 1)), self.geometry, mu, -1)
        out = v + self.kappa * acc
        if self.hermitian:
            out[:, out.shape[1] // 2:] *= -1
        return out


def _dots(a, b):
    return torch.stack([torch.vdot(x.reshape(-1), y.reshape(-1)) for x, y in zip(a, b)])


def _wide(s, like):
    return s.reshape((-1,) + (1,) * (like.dim() - 1))


def _bicgstab(op, b, tol=1e-13, steps=2000):
    x, r = torch.zeros_like(b), b.clone()
    rhat, p, v = b.clone(), torch.zeros_like(b), torch.zeros_like(b)
    one = torch.ones(b.shape[0], dtype=C128, device=b.device)
    rho, alpha, omega, bb = one, one, one, _dots(b, b).real
    for _ in range(steps):
        rho1 = _dots(rhat, r)
        p = r + _wide(rho1 / rho * alpha / omega, b) * (p - _wide(omega, b) * v)
        v = op.apply(p)
        alpha, rho = rho1 / _dots(rhat, v), rho1
        r = r - _wide(alpha, b) * v
        t = op.apply(r)
        omega = _dots(t, r) / _dots(t, t)
        x = x + _wide(alpha, b) * p + _wide(omega, b) * r
        r = r - _wide(omega, b) * t
        if float((_dots(r, r).real / bb).max()) < tol * tol:
            break
    return x


def _shifted_cg(q, b, betas, tol=1e-13, steps=5000):
    """(Q^2 + beta_k) x_k = b for all k, every system on its own."""
    s = torch.tensor(betas, dtype=torch.float64, device=b.device)
    r = b[None].repeat((len(betas),) + (1,) * b.dim())
    x, p = torch.zeros_like(r), r.clone()
    rr = _dots(r, r).real
    stop = tol * tol * rr
    for _ in range(steps):
        ap = q.apply(q.apply(p)) + _wide(s, p) * p
        a = rr / _dots(p, ap).real
        a = torch.where(rr > stop, a, torch.zeros_like(a))
        x += _wide(a, p) * p
        r -= _wide(a, p) * ap
        new = _dots(r, r).real
        p = r + _wide(torch.where(rr > stop, new / rr, torch.zeros_like(rr)), p) * p
        rr = torch.where(rr > stop, new, rr)
        if bool((rr <= stop).all()):
            break
    return x


def _fermion_force(links, geometry, kappa, alphas, xs, ys):
    u_all = _bc(links, geometry)
    nd, nc = len(geometry), links.shape[1]
    g, ns = _gammas(nd), xs.shape[1]
    gd = np.diag([1.0] * (ns // 2) + [-1.0] * (ns // 2))
    out = torch.zeros_like(links)
    for k, alpha in enumerate(alphas):
        for X, Y in ((xs[k], ys[k]), (ys[k], xs[k])):
            for mu in range(nd):
                v = torch.stack([sum(u_all[mu, i, j] * _shift(Y, geometry, mu)[:, j] for j in range(nc))
                                 for i in range(nc)], 1)
                pv = _spin(gd @ (np.eye(ns) - g[mu]), v, 0)
                px = _spin(gd @ (np.eye(ns) + g[mu]), X, 0)
                m = torch.stack([torch.stack([(X[:, i].conj() * pv[:, j] - v[:, i].conj() * px[:, j]).sum(0)
                                              for j in range(nc)]) for i in range(nc)])
                tr = sum(m[i, i] for i in range(nc)) / nc
                for i in range(nc):
                    for j in range(nc):
                        out[mu, i, j] += 0.5 * kappa * alpha * (m[j, i] - (tr if i == j else 0))
    return out


def _algebra(nc):
    """Generators with Tr T_a T_b = delta_ab / 2."""
    t = []
    for i in range(nc):
        for j in range(i + 1, nc):
            for z in (1, -1j):
                m = np.zeros((nc, nc), dtype=complex)
                m[i, j], m[j, i] = z, np.conj(z)
                t.append(m / 2)
    for i in range(1, nc):
        d = np.diag([1.0] * i + [-float(i)] + [0.0] * (nc - i - 1)).astype(complex)
        t.append(d / math.sqrt(2.0 * i * (i + 1)))
    return np.stack(t)


def _adjoint_force(links, geometry, kappa, alphas, xs, ys):
    nd, nc = len(geometry), links.shape[1]
    g, ns, t = _gammas(nd), xs.shape[1], _algebra(nc)
    na = len(t)
    gd = np.diag([1.0] * (ns // 2) + [-1.0] * (ns // 2))
    tt = torch.tensor(t, dtype=C128, device=links.device)
    comm = np.einsum("kab,ibc->kiac", t, t) - np.einsum("iab,kbc->kiac", t, t)
    ta = -2 * np.einsum("kiac,jca->kij", comm, t)
    out = torch.zeros_like(links)
    comp = 2 * torch.einsum("aij,nsjix->nsax", tt, xs), 2 * torch.einsum("aij,nsjix->nsax", tt, ys)
    for mu in range(nd):
        u = links[mu]
        w = [_mm(_mm(u, tt[b][:, :, None]), _dag(u)) for b in range(na)]
        v = torch.stack([torch.stack([2 * sum(tt[a, p, q] * w[b][q, p] for p in range(nc) for q in range(nc))
                                      for b in range(na)]) for a in range(na)])
        if mu == nd - 1:
            v[..., geometry[-1] - 1::geometry[-1]] *= -1
        c = [torch.zeros_like(u[0, 0]) for _ in range(na)]
        for k, alpha in enumerate(alphas):
            for X, Y in ((comp[0][k], comp[1][k]), (comp[1][k], comp[0][k])):
                ys1 = _shift(Y, geometry, mu)
                z = torch.stack([sum(v[a, b] * ys1[:, b] for b in range(na)) for a in range(na)], 1)
                pz = _spin(gd @ (np.eye(ns) - g[mu]), z, 0)
                px = _spin(gd @ (np.eye(ns) + g[mu]), X, 0)
                for i in range(na):
                    for j in range(na):
                        nz = [q for q in range(na) if abs(ta[q, i, j]) > 1e-14]
                        if nz:
                            m = (X[:, i].conj() * pz[:, j] - z[:, i].conj() * px[:, j]).sum(0)
                            for q in nz:
                                c[q] = c[q] + kappa * alpha * complex(ta[q, i, j]) * m
        for q in range(na):
            out[mu] += c[q] * tt[q][:, :, None]
    return out


def _staples(u, geometry, mu, skip=()):
    s = torch.zeros_like(u[mu])
    for nu in range(len(geometry)):
        if nu == mu or nu in skip:
            continue
        s += _mm(_mm(u[nu], _shift(u[mu], geometry, nu)), _dag(_shift(u[nu], geometry, mu)))
        d = _mm(_mm(_dag(u[nu]), u[mu]), _shift(u[nu], geometry, mu))
        s += _shift(d, geometry, nu, -1)
    return s


def _as_matrices(u):
    return u.permute(0, 3, 1, 2).contiguous()


def _md(links, p, geometry, beta, steps, dt):
    nc, nd = links.shape[1], len(geometry)
    u, p, lam, eps = links.clone(), p.clone(), 0.19318332275037863, dt / steps

    def kick(w):
        for mu in range(nd):
            m = _mm(u[mu], _dag(_staples(u, geometry, mu)))
            f = -0.25 * beta / nc * (_dag(m) - m)
            tr = sum(f[i, i] for i in range(nc)) / nc
            for i in range(nc):
                f[i, i] -= tr
            p[mu] += w * f

    def drift(w):
        e = torch.linalg.matrix_exp(_as_matrices(w * p)).permute(0, 2, 3, 1)
        for mu in range(nd):
            u[mu] = _mm(e[mu], u[mu].clone())

    for k in range(steps):
        kick(-lam * eps if k == 0 else -2 * lam * eps)
        drift(eps / 2)
        kick(-(1 - 2 * lam) * eps)
        drift(eps / 2)
    kick(-lam * eps)
    return u, p


def _project(m):
    """m (m^dag m)^(-1/2) / det^(1/N) for matrices (..., N, N): the polar factor by Newton's iteration."""
    n = m.shape[-1]
    for _ in range(60):
        new = 0.5 * (m + torch.linalg.inv(m).conj().transpose(-2, -1))
        done = float((new - m).abs().max()) < 1e-15
        m = new
        if done:
            break
    d = torch.linalg.det(m)
    root = torch.polar(d.abs() ** (1.0 / n), d.angle() / n)
    return m / root[..., None, None]


def _path_trace(u, geometry, steps):
    m, at = None, [0] * len(geometry)

    def link(mu):
        f = u[mu]
        for d, k in enumerate(at):
            if k:
                f = _shift(f, geometry, d, k)
        return f
    for s in steps:
        mu = abs(s) - 1
        if s > 0:
            w = link(mu)
            at[mu] += 1
        else:
            at[mu] -= 1
            w = _dag(link(mu))
        m = w if m is None else _mm(m, w)
    return sum(m[i, i] for i in range(m.shape[0]))


def _measure(links, geometry, rho):
    nd, nc, vol = len(geometry), links.shape[1], links.shape[-1]
    fat = links.clone()
    for mu in range(nd - 1):
        fat[mu] = rho / 6 * _staples(links, geometry, mu, skip=(3,)) + (1 - rho) * links[mu]
    smeared = _project(_as_matrices(fat)).permute(0, 2, 3, 1).contiguous()

    def slices(f, direction):
        keep = [d for d in range(nd) if d != direction]
        return f.reshape(geometry).sum(dim=keep)
    plaq = square = 0
    for mu in range(nd):
        for nu in range(mu + 1, nd):
            if 2 in (mu, nu):
                continue
            a, b = mu + 1, nu + 1
            plaq = plaq + _path_trace(smeared, geometry, [a, b, -a, -b])
            square = square + _path_trace(smeared, geometry, [a, a, b, b, -a, -a, -b, -b])
    count = vol // geometry[2]
    p = _path_trace(links, geometry, [4] * geometry[3])
    meson = (p * _shift(p, geometry, 1).conj()).reshape(geometry)[..., 0].sum(dim=(0, 1))
    corr = [(p * _shift(p, geometry, 2, k).conj()).mean() for k in range(geometry[2])]
    total = sum(_path_trace(links, geometry, [mu + 1, nu + 1, -(mu + 1), -(nu + 1)]).real.sum()
                for mu in range(nd) for nu in range(mu + 1, nd))
    values = [slices(plaq, 2) / count, slices(square, 2) / count, meson / (vol // (geometry[2] * geometry[3])),
              torch.stack(corr), p.mean(), total / (nd * (nd - 1) // 2 * nc * vol)]
    return smeared, [v.resolve_conj().cpu().numpy() for v in values]


def exact(case, seed):
    kind = case["kind"]
    inputs = _inputs(case, seed)
    if kind in ("solve", "lattices"):
        out = [_bicgstab(_Wilson(u, g, case["kappa"], False),
                         torch.cat([b[:, :_ns(len(g)) // 2], -b[:, _ns(len(g)) // 2:]], 1) if case["hermitian"] else b)
               for g, u, b in inputs]
        return out if kind == "lattices" else out[0]
    geometry, links, extra = inputs[0]
    if kind == "propagator":
        x = _bicgstab(_Wilson(links, geometry, case["kappa"], False), extra)
        x[:, x.shape[1] // 2:] *= -1
        keep = [d for d in range(len(geometry)) if d != case["direction"]]
        dens = (x.abs() ** 2).sum(dim=(0, 1, 2)).reshape(geometry).sum(dim=keep)
        return x, dens.to(C128).cpu().numpy()
    if kind == "rhmc_force":
        q = _Wilson(links, geometry, case["kappa"], True)
        alphas, betas = _poles(case)
        xs = _shifted_cg(q, extra, betas)
        return _fermion_force(links, geometry, case["kappa"], alphas, xs, q.apply(xs))
    if kind == "apply":
        return _Wilson(links, geometry, case["kappa"], case["hermitian"],
                       case["representation"] == "adjoint").apply(extra)
    if kind == "force":
        f = _adjoint_force if case["representation"] == "adjoint" else _fermion_force
        return f(links, geometry, case["kappa"], _poles(case)[0], extra[0], extra[1])
    if kind == "md":
        return _md(links, extra, geometry, case["beta"], int(case["steps"]), 0.1)
    return _measure(links, geometry, case["rho"])
