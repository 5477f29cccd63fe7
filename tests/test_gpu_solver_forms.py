"""The even-odd CG in each of its forms: the whole solve in one launch (small lattices) and the
launches per iteration, whichever the rule would take.  Reports say which form ran.

Tolerance: solutions to 1e-10 in the residual are within 1e-10 / s of the exact one, s >= 0.2 the
smallest singular value of D at these kappas, so two of them agree to 1e-9.
"""
import ctypes

import numpy as np
import pytest
import torch

from oracle import lym_oracle as O
from tests.test_gpu_kernel_edges import BC, cnormal, cu, make_op, smooth_links

pytestmark = pytest.mark.gpu

TOL = 1e-10


class System:
    """Links, operator and oracle of one lattice."""

    def __init__(self, rng, geom, nc, kappa=0.11, hermitian=False):
        self.u = smooth_links(rng, geom, nc)
        self.geom, self.nc, self.kappa, self.hermitian = geom, nc, kappa, hermitian
        self.op = make_op(self.u, geom, kappa, hermitian, "fundamental")
        self.ubc, self.tables = O.apply_time_bc(self.u, O.antiperiodic_field(geom, BC)), O.lookup_tables(geom)
        self.shape = (4 if len(geom) == 4 else 2, nc, int(np.prod(geom)))

    def sources(self, rng, n):
        return cnormal(rng, (n,) + self.shape)

    def residual(self, x, b):
        x = x.cpu().numpy() if isinstance(x, torch.Tensor) else x
        return np.linalg.norm(b - O.wilson_apply(self.ubc, x, self.kappa, self.hermitian, self.tables)) / np.linalg.norm(b)


def solve_on(systems, bs, xs, precision="f64", tol=TOL, max_iter=20000, **params):
    """lym_wilson_solve (one system) or lym_wilson_solve_multi on the given device buffers; the
    status and the reports."""
    from tfleonardym_b200 import _dev, _lib
    n = len(systems)
    precs = () if precision == "f64" else (precision,)
    prm = _lib.SolverParams(tol, max_iter, _lib.PREC[precision], 0.05, int(systems[0].hermitian), 8,
                            params.get("rhs_per_thread", 0), params.get("compressed_links", 0), 0, 0.0)
    counts = [int(b.shape[0]) for b in bs]
    reps = (_lib.SolverReport * sum(counts))()
    handles = [s.op.solver_gauge(precs) for s in systems]
    if n == 1:
        rc = _lib.lib().lym_wilson_solve(handles[0], systems[0].kappa, counts[0], _dev.ptr(bs[0]), _dev.ptr(xs[0]),
                                         ctypes.byref(prm), reps, _dev.stream())
    else:
        rc = _lib.lib().lym_wilson_solve_multi(
            n, (ctypes.c_void_p * n)(*[h.value for h in handles]), (ctypes.c_double * n)(*[s.kappa for s in systems]),
            None, (ctypes.c_int * n)(*counts), (ctypes.c_void_p * n)(*[b.data_ptr() for b in bs]),
            (ctypes.c_void_p * n)(*[x.data_ptr() for x in xs]), ctypes.byref(prm), reps, _dev.stream())
    return rc, list(reps)


def one_launch(reports):
    return all(r.kernel_launches == 1 for r in reports)


def test_solutions_over_sources(cuda_device):
    """x may cover b: exactly, shifted by one right-hand side, or those of another lattice.  A
    shifted one goes launch by launch, which reads every source first."""
    rng = np.random.default_rng(31)
    s = System(rng, (8, 12), 2)
    b = s.sources(rng, 3)
    buf = cu(b)
    rc, reps = solve_on([s], [buf], [buf])
    assert rc == 0 and one_launch(reps)
    assert max(s.residual(buf[i], b[i]) for i in range(3)) < TOL
    for b_at, x_at in ((0, 1), (1, 0)):
        buf = torch.zeros((4,) + s.shape, dtype=torch.complex128, device="cuda")
        buf[b_at:b_at + 3] = cu(b)
        rc, reps = solve_on([s], [buf[b_at:b_at + 3]], [buf[x_at:x_at + 3]])
        assert rc == 0 and not one_launch(reps)
        assert max(s.residual(buf[x_at + i], b[i]) for i in range(3)) < TOL
    systems = [System(rng, (8, 12), 2, 0.10), System(rng, (6, 16), 2, 0.12)]  # 96 sites each
    bs = [t.sources(rng, 2) for t in systems]
    bufs = [cu(t) for t in bs]
    rc, reps = solve_on(systems, bufs, bufs)
    assert rc == 0 and one_launch(reps)
    for t, x, c in zip(systems, bufs, bs):
        assert max(t.residual(x[i], c[i]) for i in range(2)) < TOL
    bufs = [cu(t) for t in bs]
    rc, reps = solve_on(systems, bufs, bufs[::-1])
    assert rc == 0 and not one_launch(reps)
    for t, x, c in zip(systems, bufs[::-1], bs):
        assert max(t.residual(x[i], c[i]) for i in range(2)) < TOL
