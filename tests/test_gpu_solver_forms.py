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


class LargeSystem:
    """Links made on the device; residuals by the operator, whose own tests hold it to the oracle."""

    def __init__(self, geom, nc, kappa=0.11, hermitian=False):
        from tfleonardym_b200 import boundary_conditions as bc
        from tfleonardym_b200 import dirac, smearing
        from tfleonardym_b200 import lattice as lt
        vol = int(np.prod(geom))
        gen = torch.Generator(device="cuda")
        gen.manual_seed(vol + nc)
        self.gen, self.shape = gen, (4 if len(geom) == 4 else 2, nc, vol)
        self.kappa, self.hermitian = kappa, hermitian
        u = 0.3 * self.normal((len(geom), nc, nc, vol))
        for i in range(nc):
            u[:, i, i] += 1
        cfg = lt.Configuration(smearing.unitary_sqrt_projection(u), geom, nc, len(geom))
        self.op = dirac.DiracWilsonOperator(cfg, kappa, hermitian, representation="fundamental",
                                            boundary_condition_provider=bc.factor_provider(BC))

    def normal(self, shape):
        return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=self.gen, dtype=torch.float64,
                                                 device="cuda"))

    def residual(self, x, b):
        return float(torch.linalg.vector_norm(b - self.op.apply(x)) / torch.linalg.vector_norm(b))


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


@pytest.mark.parametrize("precision", ["f32", "f16", "bf16"])
def test_launches_of_the_resident_form_are_bounded(cuda_device, precision):
    """A tolerance that is never met runs to max_iter over several launches.  600 systems on
    8 x 8 (one block of 64 threads each, two waves of blocks, 4096 iterations a launch) against
    the same right-hand side alone (8192 a launch): the same steps, bit for bit."""
    rng = np.random.default_rng(7)
    systems = [System(rng, (8, 8), 2, k) for k in (0.10, 0.12)]
    bs = [s.sources(rng, 300) for s in systems]
    xs = [torch.empty_like(cu(b)) for b in bs]
    rc, reps = solve_on(systems, [cu(b) for b in bs], xs, precision, tol=1e-17, max_iter=5000)
    assert rc != 0 and {r.kernel_launches for r in reps} == {2} and {r.iterations for r in reps} == {5000}
    alone = torch.empty((1,) + systems[1].shape, dtype=torch.complex128, device="cuda")
    for k in (0, 299):
        rc, reps1 = solve_on(systems[1:], [cu(bs[1][k:k + 1])], [alone], precision, tol=1e-17, max_iter=5000)
        assert rc != 0 and one_launch(reps1) and reps1[0].iterations == 5000
        assert torch.equal(alone[0], xs[1][k])
        assert reps1[0].true_residual == reps[300 + k].true_residual
        assert reps1[0].reliable_updates == reps[300 + k].reliable_updates
        if precision != "bf16":  # whose 8 bits lose the directions: FP64 updates hold the others near rounding
            assert systems[1].residual(alone[0], bs[1][k]) < 1e-13
    rc, reps1 = solve_on(systems[1:], [cu(bs[1][:1])], [alone], precision, tol=1e-17, max_iter=20000)
    assert rc != 0 and reps1[0].kernel_launches == 3 and reps1[0].iterations == 20000


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_solves_that_converge_over_several_launches(cuda_device, precision):
    """1024 systems in clusters of 8 x 128 with two sites per thread: 28 waves, 146 iterations a launch.
    The same right-hand sides in a call of 40 (the same clusters, two waves, 2048 a launch) give the
    same bits.  Residuals are formed to 1e-16, 1 % of this tolerance at most."""
    tol = 1e-13
    systems = [LargeSystem((16, 16, 16), 2, k) for k in (0.18, 0.12)]
    bs = [s.normal((512,) + s.shape) for s in systems]
    xs = [torch.empty_like(b) for b in bs]
    rc, reps = solve_on(systems, bs, xs, precision, tol)
    assert rc == 0 and reps[0].kernel_launches > 1 and max(r.iterations for r in reps[:512]) > 146
    few = torch.empty_like(bs[0][:40])
    rc, reps40 = solve_on(systems[:1], [bs[0][:40]], [few], precision, tol)
    assert rc == 0 and one_launch(reps40)
    assert torch.equal(few, xs[0][:40])
    assert [r.iterations for r in reps40] == [r.iterations for r in reps[:40]]
    assert [r.true_residual for r in reps40] == [r.true_residual for r in reps[:40]]
    for s, b, x in zip(systems, bs, xs):
        assert max(s.residual(x[i], b[i]) for i in (0, 200, 511)) < 1.01 * tol


@pytest.mark.parametrize("tiled", [0, 1])
@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
def test_solves_that_cannot_go_on_end(cuda_device, precision, tiled):
    """A source that is not finite takes no step; the other right-hand sides converge and the call
    returns, in both forms and on several lattices.  So does one whose residual falls to zero short
    of its target."""
    from tfleonardym_b200 import _lib
    rng = np.random.default_rng(3)
    systems = [System(rng, g, 2) for g in ((8, 12), (6, 10))]
    bs = [s.sources(rng, 3) for s in systems]
    bs[0][2, 0, 0, 5] = np.nan
    bs[1][0, 1, 1, 7] = np.nan
    want = [0, 0, _lib.LYM_ERR_NOT_CONVERGED, _lib.LYM_ERR_NOT_CONVERGED, 0, 0]
    for n in (1, 2):
        xs = [torch.empty_like(cu(b)) for b in bs[:n]]
        rc, reps = solve_on(systems[:n], [cu(b) for b in bs[:n]], xs, precision, rhs_per_thread=tiled)
        assert rc == _lib.LYM_ERR_NOT_CONVERGED and [r.status for r in reps] == want[:3 * n]
        for s, b, x, st in zip(systems, bs, xs, (want[:3], want[3:])):
            assert max(s.residual(x[i], b[i]) for i in range(3) if st[i] == 0) < TOL
    x = torch.empty_like(cu(bs[0][:1]))
    rc, reps = solve_on(systems[:1], [cu(bs[0][:1])], [x], precision, tol=1e-30, max_iter=2000, rhs_per_thread=tiled)
    assert rc == _lib.LYM_ERR_NOT_CONVERGED and reps[0].iterations <= 2000


# blocks: 81 each; three waves of two per SM instead of two of three in 4D SU(3) up to 888 (and from 1185),
# the usual form between; SU(2) from 593 on
@pytest.mark.parametrize("nc,nrhs", [(3, 7), (3, 8), (3, 11), (3, 12), (3, 16), (2, 12)])
def test_fp64_solves_of_both_occupancies(cuda_device, nc, nrhs):
    s = LargeSystem((12, 12, 12, 12), nc)
    b = s.normal((nrhs,) + s.shape)
    x = torch.empty_like(b)
    rc, reps = solve_on([s], [b], [x], "f64")
    assert rc == 0 and not one_launch(reps)
    assert max(s.residual(x[i], b[i]) for i in range(nrhs)) < TOL


def test_hop_alone_after_a_one_launch_solve(cuda_device):
    """lym_dslash_eo on a workspace that only one-launch solves have used: picks a hop form as a
    launch-by-launch solve does, and the workspace solves on in both forms."""
    from tfleonardym_b200 import _dev, _lib
    rng = np.random.default_rng(14)
    s = System(rng, (4, 4, 4, 8), 3)
    b = s.sources(rng, 4)
    for precision in ("f64", "f32", "f16"):
        x = torch.empty_like(cu(b))
        for tiled in (0, 1, 0):
            rc, reps = solve_on([s], [cu(b)], [x], precision, rhs_per_thread=tiled)
            assert rc == 0 and one_launch(reps) == (not tiled)
            assert max(s.residual(x[i], b[i]) for i in range(4)) < TOL
            handle = s.op.solver_gauge(() if precision == "f64" else (precision,))
            assert _lib.lib().lym_dslash_eo(handle, _lib.PREC[precision], 4, 3, _dev.stream()) == 0
        assert _lib.lib().lym_dslash_eo(handle, _lib.PREC[precision], 999, 1, _dev.stream()) == _lib.LYM_ERR_BAD_ARG


@pytest.mark.parametrize("precision", ["f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("geoms,nc,herm", [([(8, 8), (4, 6), (32, 34)], 2, False), ([(6, 10), (12, 16)], 3, True),
                                           ([(4, 4, 4, 4), (2, 4, 6, 8), (4, 4, 4, 10)], 3, False),
                                           ([(4, 4, 4, 4), (2, 6, 4, 8)], 2, True),
                                           ([(4, 4, 4), (8, 6, 4)], 3, False), ([(6, 4, 4), (16, 16, 16)], 2, False)])
def test_lattices_launch_by_launch(cuda_device, geoms, nc, herm, precision):
    """The kernels over all lattices of a call, which lists of small lattices reach only with a
    forced tile: FP32 with the compressed links of SU(N) fields, FP16 with the mixed-precision hop
    (2 and 4 dimensions).  The one-launch form solves the same systems."""
    rng = np.random.default_rng(len(geoms) + nc)
    systems = [System(rng, g, nc, 0.10 + 0.01 * k, herm) for k, g in enumerate(geoms)]
    bs = [s.sources(rng, 1 + 2 * k) for k, s in enumerate(systems)]
    for tiled in (1, 0, 1):
        xs = [torch.empty_like(cu(b)) for b in bs]
        rc, reps = solve_on(systems, [cu(b) for b in bs], xs, precision, rhs_per_thread=tiled)
        assert rc == 0 and one_launch(reps) == (not tiled)
        assert {r.compressed_links for r in reps} == {int(tiled and precision == "f32")}
        assert {r.mixed_fma for r in reps} == {int(tiled and precision == "f16" and len(geoms[0]) != 3)}
        for s, b, x in zip(systems, bs, xs):
            assert max(s.residual(x[i], b[i]) for i in range(len(b))) < TOL


@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
def test_one_workspace_in_both_forms(cuda_device, precision):
    """A workspace that the one-launch form left with more sources than a launch-by-launch solve
    has: the padding starts empty again, so the solve takes the launches and gives the bits of one
    on fresh links."""
    rng = np.random.default_rng(12)
    s = System(rng, (4, 4, 4, 8), 3)
    b = cu(s.sources(rng, 8))

    def solve(system, n, tiled):
        x = torch.empty_like(b[:n])
        rc, reps = solve_on([system], [b[:n]], [x], precision, rhs_per_thread=tiled)
        assert rc == 0 and one_launch(reps) == (not tiled)
        return x, reps[0].kernel_launches

    for n, tiled in ((8, 0), (5, 1), (7, 0), (6, 1), (8, 1), (5, 0), (5, 1), (3, 0), (4, 0), (3, 1)):
        x, launches = solve(s, n, tiled)
        fresh = System.__new__(System)
        fresh.__dict__.update(s.__dict__)
        fresh.op = make_op(s.u, s.geom, s.kappa, False, "fundamental")
        y, fresh_launches = solve(fresh, n, tiled)
        assert torch.equal(x, y) and launches == fresh_launches, (n, tiled)
        assert max(s.residual(x[i], b[i].cpu().numpy()) for i in range(n)) < TOL


@pytest.mark.parametrize("geom,nc", [((4, 4, 4, 8), 3), ((4, 2, 4, 6), 2), ((8, 12), 3), ((4, 6, 4), 3)])
@pytest.mark.parametrize("precision", ["f32", "f16", "bf16"])
def test_compressed_links(cuda_device, geom, nc, precision):
    rng = np.random.default_rng(nc)
    s = System(rng, geom, nc)
    b = s.sources(rng, 4)
    for tile in (1, 2, 4):
        x = torch.empty_like(cu(b))
        rc, reps = solve_on([s], [cu(b)], [x], precision, rhs_per_thread=tile, compressed_links=1)
        assert rc == 0 and {(r.rhs_per_thread, r.compressed_links) for r in reps} == {(tile, 1)}
        assert max(s.residual(x[i], b[i]) for i in range(4)) < TOL


# the sizes on either side of the one-launch rule, by its tables; 4D SU(3) FP64 takes 12 right-hand sides
# up to 2048 sites per parity
@pytest.mark.parametrize("geom,nc,precision,nrhs,resident",
                         [((64, 128), 2, "f64", 1, True), ((64, 130), 2, "f64", 1, False),
                          ((128, 128), 3, "f32", 2, True), ((128, 130), 3, "f32", 2, False),
                          ((16, 16, 16), 3, "f64", 1, True), ((16, 16, 18), 3, "f64", 1, False),
                          ((16, 16, 18), 3, "f16", 1, True), ((8, 8, 8, 8), 2, "f64", 12, True),
                          ((8, 8, 8, 8), 2, "f64", 13, False), ((8, 8, 12, 16), 3, "f32", 3, False),
                          ((8, 8, 12, 16), 2, "bf16", 2, False), ((8, 8, 8, 8), 3, "f16", 25, False)])
def test_the_form_the_rule_takes(cuda_device, geom, nc, precision, nrhs, resident):
    """Which form runs, and its answer; where it is not the resident one, with the tile that the
    autotuner picks (compressed links among the FP32 and BF16 candidates)."""
    rng = np.random.default_rng(int(np.prod(geom)))
    s = System(rng, geom, nc)
    b = s.sources(rng, nrhs)
    x = torch.empty_like(cu(b))
    rc, reps = solve_on([s], [cu(b)], [x], precision)
    assert rc == 0 and one_launch(reps) == resident
    for i in {0, nrhs // 2, nrhs - 1}:
        assert s.residual(x[i], b[i]) < TOL


# more than 64 MB of links in the precision of the hop and several tiles: the right-hand side is the
# fast index of the grid (in every hop of the FP64 solve, in the FP64 updates of the others, in the sloppy
# hops from 24^3 x 16 in FP32 and 24^3 x 32 in FP16 on); 16^3 x 28 lies below in FP64
@pytest.mark.parametrize("geom,nc,precision,nrhs,tile", [((16, 16, 16, 28), 3, "f64", 2, 0),
                                                         ((16, 16, 16, 32), 3, "f64", 2, 0),
                                                         ((16, 16, 16, 30), 3, "f64", 3, 0),
                                                         ((16, 16, 16, 32), 3, "f32", 4, 2),
                                                         ((24, 24, 24, 16), 3, "f32", 4, 2),
                                                         ((24, 24, 24, 16), 3, "f32", 8, 4),
                                                         ((24, 24, 24, 32), 3, "f16", 4, 1),
                                                         ((24, 24, 24, 32), 3, "f16", 4, 0)])
def test_grids_with_the_right_hand_side_fastest(cuda_device, geom, nc, precision, nrhs, tile):
    s = LargeSystem(geom, nc)
    b = s.normal((nrhs,) + s.shape)
    b *= torch.arange(1, nrhs + 1, device="cuda")[:, None, None, None]  # sources that cannot be taken for each other
    x = torch.empty_like(b)
    rc, reps = solve_on([s], [b], [x], precision, rhs_per_thread=tile)
    assert rc == 0 and (not tile or reps[0].rhs_per_thread == tile)
    assert max(s.residual(x[i], b[i]) for i in range(nrhs)) < TOL


@pytest.mark.parametrize("geom,nc,precision,nrhs", [((16, 16, 16), 2, "f64", 40), ((16, 16, 16), 2, "f32", 64),
                                                    ((32, 66), 3, "f64", 64), ((32, 66), 3, "f16", 40),
                                                    ((8, 8, 8, 8), 3, "f32", 24)])
def test_more_clusters_than_fit_at_once(cuda_device, geom, nc, precision, nrhs):
    """Above 1024 sites per parity with more right-hand sides than clusters of 8 x 256 threads fit:
    clusters of 8 x 128."""
    s = LargeSystem(geom, nc)
    b = s.normal((nrhs,) + s.shape)
    x = torch.empty_like(b)
    rc, reps = solve_on([s], [b], [x], precision)
    assert rc == 0 and one_launch(reps)
    assert max(s.residual(x[i], b[i]) for i in range(nrhs)) < TOL


# blocks of the operator kernels: 324 and 392 (one wave of three per SM instead of two of two) and 640 (two
# instead of three); the usual form for 314 in 2D SU(2), 768 in 4D SU(3) and 512
@pytest.mark.parametrize("geom,nc", [((12, 12, 12, 24), 3), ((12, 12, 12, 24), 2), ((224, 224), 2), ((200, 200), 2),
                                     ((16, 16, 16, 20), 3), ((16, 16, 16, 24), 3), ((16, 16, 16, 16), 3)])
def test_multishift_of_both_occupancies(cuda_device, geom, nc):
    from tfleonardym_b200 import dirac, dirac_solver
    s = LargeSystem(geom, nc, hermitian=True)
    b = s.normal(s.shape)
    shifts = [0.05, 0.4, 2.0]
    xs = dirac_solver.multishift_cg(5000, TOL, precision="f64").solve(dirac.SquareOperator(s.op), b, shifts)
    for x, shift in zip(xs, shifts):
        res = b - s.op.apply(s.op.apply(x)) - shift * x
        assert float(torch.linalg.vector_norm(res) / torch.linalg.vector_norm(b)) < TOL * 1.01
