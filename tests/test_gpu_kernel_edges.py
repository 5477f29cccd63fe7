"""Kernels at the sizes where their work split can go wrong: site counts that fill no
warp or block, one-site extents, links that are not unitary, spinors with a trace part,
a complex boundary factor.  Against the CPU oracle.

Tolerance: every output is a sum of at most a few hundred FP64 products of unit-size
numbers; 1e-13 relative (norm of the difference over norm) leaves a factor of ten over
the rounding of the longest of them.
"""
import numpy as np
import pytest
import torch

from oracle import lym_oracle as O
from tests.conftest import relerr

pytestmark = pytest.mark.gpu

TOL = 1e-13
BC = -0.6 + 0.8j


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def cnormal(rng, shape):
    return rng.normal(size=shape) + 1j * rng.normal(size=shape)


def links(rng, geom, nc, unitary=True):
    x = cnormal(rng, (len(geom), nc, nc, int(np.prod(geom))))
    return O.unitary_sqrt_projection(x) if unitary else x


def make_op(u, geom, kappa, hermitian, representation):
    from tfleonardym_b200 import boundary_conditions as bc
    from tfleonardym_b200 import dirac
    from tfleonardym_b200 import lattice as lt
    cfg = lt.Configuration(cu(u), geom, u.shape[1], len(geom))
    bc.set_antiperiodic_field_in_t_direction(geom, BC)
    return dirac.DiracWilsonOperator(cfg, kappa, hermitian, representation=representation,
                                     boundary_condition_provider=bc.factor_provider(BC))


@pytest.mark.parametrize("geom,nc,unitary", [((3, 5), 2, True), ((1, 11), 3, False), ((2, 1, 3, 3), 3, True),
                                             ((3, 1, 2, 7), 2, False), ((1, 2, 2, 4), 3, False)])
def test_adjoint_operator_and_force_on_ragged_lattices(cuda_device, geom, nc, unitary):
    rng = np.random.default_rng(int(np.prod(geom)) + nc)
    nd, vol, kappa = len(geom), int(np.prod(geom)), 0.11
    ns = 4 if nd == 4 else 2
    u = links(rng, geom, nc, unitary)
    tables, field = O.lookup_tables(geom), O.antiperiodic_field(geom, BC)
    x, y = cnormal(rng, (3, ns, nc, nc, vol)), cnormal(rng, (3, ns, nc, nc, vol))
    alphas = [0.7, -1.3, 0.2]
    v = O.adjoint_links(u, field)
    for herm in (False, True):
        op = make_op(u, geom, kappa, herm, "adjoint")
        out = op.apply(cu(x)).cpu().numpy()
        for k in range(3):
            ref = O.wilson_apply_adjoint(O.apply_time_bc(u, field), u, x[k], kappa, herm, tables)
            assert relerr(out[k], ref) < TOL, (herm, k)
        for symmetric in (False, True):
            ref = np.zeros((nd, nc, nc, vol), complex)
            for k, a in enumerate(alphas):
                ref += a * O.lie_derivative_adjoint(v, x[k], y[k], kappa, herm, tables)
                if symmetric:
                    ref += a * O.lie_derivative_adjoint(v, y[k], x[k], kappa, herm, tables)
            start = cnormal(rng, ref.shape)
            f = op.accumulate_force(cu(start), alphas, cu(x), cu(y), symmetric=symmetric, scale=0.5)
            assert relerr(f.cpu().numpy(), start + 0.5 * ref) < TOL, (herm, symmetric)


@pytest.mark.parametrize("geom,nc,unitary", [((5, 7), 3, False), ((33, 1), 2, True), ((3, 2, 3, 5), 3, False),
                                             ((1, 2, 4, 4), 2, True), ((3, 3, 1, 11), 3, True)])
def test_fundamental_force_on_ragged_lattices(cuda_device, geom, nc, unitary):
    rng = np.random.default_rng(int(np.prod(geom)) + nc)
    nd, vol, kappa = len(geom), int(np.prod(geom)), 0.13
    ns = 4 if nd == 4 else 2
    u = links(rng, geom, nc, unitary)
    tables, ubc = O.lookup_tables(geom), O.apply_time_bc(u, O.antiperiodic_field(geom, BC))
    x, y = cnormal(rng, (3, ns, nc, vol)), cnormal(rng, (3, ns, nc, vol))
    alphas = [0.7, -1.3, 0.2]
    for herm in (False, True):
        op = make_op(u, geom, kappa, herm, "fundamental")
        for symmetric in (False, True):
            ref = np.zeros((nd, nc, nc, vol), complex)
            for k, a in enumerate(alphas):
                ref += a * O.lie_derivative(ubc, x[k], y[k], kappa, herm, tables)
                if symmetric:
                    ref += a * O.lie_derivative(ubc, y[k], x[k], kappa, herm, tables)
            start = cnormal(rng, ref.shape)
            f = op.accumulate_force(cu(start), alphas, cu(x), cu(y), symmetric=symmetric, scale=0.5)
            assert relerr(f.cpu().numpy(), start + 0.5 * ref) < TOL, (herm, symmetric)


GEOMETRIES = [(7, 3), (2, 37), (3, 5, 2), (3, 1, 5, 7), (4, 3, 2, 33)]


@pytest.mark.parametrize("geom", GEOMETRIES)
@pytest.mark.parametrize("nc", [2, 3])
def test_plaquette_staples_and_paths_on_ragged_lattices(cuda_device, geom, nc):
    from tfleonardym_b200 import gauge_action, measurements, staples
    from tfleonardym_b200 import lattice as lt
    rng = np.random.default_rng(int(np.prod(geom)) * nc)
    nd = len(geom)
    u = links(rng, geom, nc, unitary=False)
    tables = O.lookup_tables(geom)
    cfg = lt.Configuration(cu(u), geom, nc, nd)
    re, im = gauge_action.plaquette_trace_sum(cfg)
    ref = O.plaquette_trace_sum(u, tables)
    assert abs(complex(re, im) - ref) < TOL * np.sum(np.abs(u) ** 4)
    for nodir in [-1] + list(range(nd)):
        st = staples.get_staple_sums(cfg, nodir).cpu().numpy()
        assert relerr(st, O.staples(u, tables, nodir if nodir >= 0 else None)) < TOL
    f = gauge_action.yang_mills(cfg, 5.5).force().cpu().numpy()
    assert relerr(f, O.gauge_force(u, 5.5, tables)) < TOL
    # unit-size links, so that no length of a path overflows its tolerance
    u = links(rng, geom, nc)
    cfg = lt.Configuration(cu(u), geom, nc, nd)
    paths = [[], [1], [-2], [2, -1], [1, 2, -1, -2], [nd, nd, -1, nd, 2], [1] * geom[0], [nd] * geom[-1],
             [nd] * (geom[-1] + 1), [-nd] * geom[-1]]
    for steps in paths:
        got = measurements.path_field(cfg, steps).cpu().numpy()
        if steps:
            assert relerr(got, O.path_trace(u, tables, steps)) < TOL * max(1, len(steps)), steps
            m = measurements.path_field(cfg, steps, trace=False).cpu().numpy()
            assert relerr(m, O.path_product(u, tables, steps)) < TOL * max(1, len(steps)), steps
        else:
            assert np.all(got == nc)


@pytest.mark.parametrize("geom", GEOMETRIES + [(6, 8, 4, 10)])
def test_slice_sums_and_shifted_products(cuda_device, geom):
    from tfleonardym_b200 import _dev, _lib, measurements
    from tfleonardym_b200 import lattice as lt
    rng = np.random.default_rng(int(np.prod(geom)))
    vol = int(np.prod(geom))
    f = cnormal(rng, (vol,))
    cfg = lt.Configuration(cu(links(rng, geom, 2)), geom, 2, len(geom))
    grid = f.reshape(geom)
    for d in range(len(geom)):
        others = tuple(k for k in range(len(geom)) if k != d)
        scale = TOL * np.sum(np.abs(f))
        assert np.max(np.abs(measurements._slice_sums(cfg, cu(f), d) - grid.sum(axis=others))) < scale
        for m in others:
            ref = grid.take([0], axis=m).sum(axis=others)
            assert np.max(np.abs(measurements._slice_sums(cfg, cu(f), d, m) - ref)) < scale
        ref = np.array([np.vdot(np.roll(grid, -k, axis=d), grid) for k in range(geom[d])])
        assert np.max(np.abs(measurements._shift_dots(cfg, cu(f), d) - ref)) < TOL * np.sum(np.abs(f) ** 2)
        for adjoint in (0, 1):
            v = cnormal(rng, (3, 2, 2, 2, vol)) if adjoint else cnormal(rng, (3, 2, 3, vol))
            w = np.swapaxes(v, 2, 3) if adjoint else v
            ref = (np.conj(v) * w).reshape((-1, vol)).sum(0).reshape(geom).sum(axis=others)
            out = torch.empty(2 * geom[d], dtype=torch.float64, device="cuda")
            x = cu(v)
            _lib.check(_lib.lib().lym_timeslice_sums(lt.get_lattice(geom).handle, d, 3, 2, 2 if adjoint else 3, adjoint,
                                                     _dev.ptr(x), _dev.ptr(out), _dev.stream()), "lym_timeslice_sums")
            o = out.cpu().numpy()
            assert np.max(np.abs(o[0::2] + 1j * o[1::2] - ref)) < TOL * np.sum(np.abs(v) ** 2)


def smooth_links(rng, geom, nc, spread=0.3):
    x = spread * cnormal(rng, (len(geom), nc, nc, int(np.prod(geom))))
    for i in range(nc):
        x[:, i, i] += 1
    return O.unitary_sqrt_projection(x)


# sites per parity: one block of 64 (2, 8, 64) and of 256 threads (256), the first cluster
# (272), full clusters of 128 (1024) and the first of 256 threads (1056), two sites per
# thread (4096), and the last sizes of the rule (8192 in reduced precisions, 2D)
SOLVE_SHAPES = [((2, 2), 2), ((2, 2, 2, 2), 3), ((8, 16), 3), ((16, 32), 2), ((16, 34), 2), ((32, 64), 2),
                ((32, 66), 3), ((64, 128), 2), ((128, 128), 2), ((8, 8, 8), 2), ((6, 10, 10), 3), ((16, 16, 16), 2),
                ((4, 4, 4, 8), 2), ((4, 4, 6, 8), 3), ((8, 8, 8, 8), 3)]


@pytest.mark.parametrize("precision", ["f64", "f32", "f16", "bf16"])
@pytest.mark.parametrize("geom,nc", SOLVE_SHAPES)
def test_solve_on_small_lattices(cuda_device, geom, nc, precision):
    """True residuals by the oracle below the target; the solutions of the launch-per-kernel
    form (a forced tile) to the accuracy both targets leave: each is within tol / s of the
    exact one, s >= 0.2 the smallest singular value of D at this kappa, so 1e-9 apart."""
    from tfleonardym_b200 import dirac_solver
    rng = np.random.default_rng(int(np.prod(geom)) + nc)
    nd, vol, kappa, tol = len(geom), int(np.prod(geom)), 0.11, 1e-10
    ns = 4 if nd == 4 else 2
    u = smooth_links(rng, geom, nc)
    ubc, tables = O.apply_time_bc(u, O.antiperiodic_field(geom, BC)), O.lookup_tables(geom)
    b = cnormal(rng, (3, ns, nc, vol))
    for herm in ([False] if nd == 3 else [False, True]):
        op = make_op(u, geom, kappa, herm, "fundamental")
        solver = dirac_solver.conjugate_gradient(tol=tol, precision=precision, delta=0.05)
        x = solver.solve(op, cu(b))
        tiled = dirac_solver.conjugate_gradient(tol=tol, precision=precision, delta=0.05, rhs_per_thread=1)
        y = tiled.solve(op, cu(b))
        for i in range(3):
            res = np.linalg.norm(b[i] - O.wilson_apply(ubc, x[i].cpu().numpy(), kappa, herm, tables))
            assert res < tol * np.linalg.norm(b[i]), (herm, i, solver.reports[i])
            assert solver.reports[i]["status"] == 0 and abs(solver.reports[i]["true_residual"] * np.linalg.norm(b[i])
                                                            - res) < 0.01 * tol * np.linalg.norm(b[i])
            assert relerr(x[i].cpu().numpy(), y[i].cpu().numpy()) < 10 * tol
        alone = solver.solve(op, cu(b[1]))
        assert relerr(alone.cpu().numpy(), x[1].cpu().numpy()) < 10 * tol


def test_solve_on_small_lattices_stops(cuda_device):
    """Zero sources, the iteration limit and sources that are not finite end the solve."""
    from tfleonardym_b200 import _lib, dirac_solver
    rng = np.random.default_rng(5)
    geom, nc = (8, 12), 2
    op = make_op(smooth_links(rng, geom, nc), geom, 0.12, True, "fundamental")
    b = cnormal(rng, (3, 2, nc, 96))
    b[1] = 0
    for precision in ("f64", "f32", "f16"):
        solver = dirac_solver.conjugate_gradient(max_steps=3, tol=1e-12, precision=precision)
        x = solver.solve(op, cu(b)).cpu().numpy()
        assert [r["iterations"] for r in solver.reports] == [3, 0, 3]
        assert [r["status"] for r in solver.reports] == [_lib.LYM_ERR_NOT_CONVERGED, 0, _lib.LYM_ERR_NOT_CONVERGED]
        assert np.all(x[1] == 0) and np.all(np.isfinite(x))
        c = b.copy()
        c[2, 0, 0, 5] = np.nan
        solver = dirac_solver.conjugate_gradient(tol=1e-10, precision=precision)
        x = solver.solve(op, cu(c)).cpu().numpy()
        assert [r["status"] for r in solver.reports] == [0, 0, _lib.LYM_ERR_NOT_CONVERGED]
        assert np.all(np.isfinite(x[:2]))


@pytest.mark.parametrize("precision", ["f64", "f32", "f16"])
@pytest.mark.parametrize("geoms,nc", [([(8, 8), (4, 6), (32, 34), (2, 4)], 2),
                                      ([(4, 4, 4, 4), (2, 4, 6, 8), (4, 4, 4, 10)], 3),
                                      ([(4, 4, 4), (18, 16, 16), (8, 6, 4)], 2)])
def test_lattices_of_uneven_sizes_together(cuda_device, geoms, nc, precision):
    """Every lattice's own kappa, tolerance and number of sources; the last list has a lattice
    above the resident form's limit, so it runs launch by launch."""
    from tfleonardym_b200 import dirac_solver
    rng = np.random.default_rng(len(geoms) + nc)
    ops, bs, refs = [], [], []
    for k, g in enumerate(geoms):
        nd, vol = len(g), int(np.prod(g))
        u = smooth_links(rng, g, nc)
        kappa = 0.10 + 0.01 * k
        ops.append(make_op(u, g, kappa, False, "fundamental"))
        bs.append(cnormal(rng, (1 + k, 4 if nd == 4 else 2, nc, vol)))
        refs.append((O.apply_time_bc(u, O.antiperiodic_field(g, BC)), kappa, O.lookup_tables(g)))
    tols = [1e-10, 1e-9, 1e-11, 1e-10][:len(geoms)]
    xs, reports = dirac_solver.solve_lattices(ops, [cu(b) for b in bs], precision=precision, tols=tols)
    for k in range(len(geoms)):
        for i in range(bs[k].shape[0]):
            res = np.linalg.norm(bs[k][i] - O.wilson_apply(refs[k][0], xs[k][i].cpu().numpy(), refs[k][1], False,
                                                           refs[k][2])) / np.linalg.norm(bs[k][i])
            assert res < tols[k], (k, i, reports[k][i])
            assert reports[k][i]["status"] == 0


# the last two lie on either side of the size from which 4D SU(3) runs blocks of eight warps
@pytest.mark.parametrize("geom,nc", [((7, 3), 3), ((3, 5, 2), 2), ((4, 3, 2, 33), 2), ((3, 1, 5, 7), 3),
                                     ((7, 9, 28, 32), 3), ((7, 9, 30, 31), 3)])
def test_kick_and_drift_in_one_pass(cuda_device, geom, nc):
    """Momenta and links after one gauge kick and drift, the force alone and one smearing step.
    Momenta and forces of order one per entry: exp(0.1 P) takes a few dozen more products; links
    near the identity keep the projection well conditioned."""
    from tfleonardym_b200 import gauge_action, smearing
    from tfleonardym_b200 import lattice as lt
    rng = np.random.default_rng(int(np.prod(geom)) + nc)
    u, beta, eps_p, eps_u = smooth_links(rng, geom, nc, spread=0.05), 5.5, -0.15, 0.1
    x = cnormal(rng, u.shape)
    p = 0.5 * (x - np.conj(np.swapaxes(x, 1, 2)))
    p -= np.einsum("miiv->mv", p)[:, None, None] * (np.eye(nc) / nc)[None, :, :, None]
    tables = O.lookup_tables(geom)
    force = O.gauge_force(u, beta, tables)
    kicked = O.update_momenta(p, force, eps_p)
    action = gauge_action.yang_mills(lt.Configuration(cu(u), geom, nc, len(geom)), beta)
    given = cu(p)
    p_out, u_out = action.kick_and_drift(given, eps_p, eps_u)
    assert relerr(p_out.cpu().numpy(), kicked) < TOL
    assert relerr(u_out.cpu().numpy(), O.update_link_field(u, kicked, eps_u)) < TOL
    assert np.array_equal(given.cpu().numpy(), p)
    assert np.array_equal(action.cfg.gauge_field.cpu().numpy(), u)
    assert relerr(action.force().cpu().numpy(), force) < TOL
    fat = smearing.ape_smearing(action.cfg, 0.3, len(geom) - 1)
    fat = getattr(fat, "gauge_field", fat)
    assert relerr(fat.cpu().numpy(), O.ape_smearing(u, tables, 0.3, len(geom) - 1)) < TOL


# sites per parity: less than one block, ragged blocks; 23 and 24 sources on 25 blocks lie on either
# side of the line (592 blocks) to the form with three blocks per SM
@pytest.mark.parametrize("geom,nc,nrhs", [((2, 2), 3, 2), ((10, 16), 2, 3), ((6, 6, 10), 3, 2), ((6, 22), 2, 1),
                                          ((4, 4, 4, 6), 3, 3), ((2, 10, 6, 10), 2, 5), ((8, 8, 10, 10), 2, 23),
                                          ((8, 8, 10, 10), 2, 24)])
def test_fp64_solves_launch_by_launch(cuda_device, geom, nc, nrhs):
    """True residuals by the oracle; a forced tile keeps the solve out of the one-launch form."""
    from tfleonardym_b200 import dirac_solver
    rng = np.random.default_rng(int(np.prod(geom)) + nc + nrhs)
    nd, vol, kappa, tol = len(geom), int(np.prod(geom)), 0.11, 1e-10
    u = smooth_links(rng, geom, nc)
    ubc, tables = O.apply_time_bc(u, O.antiperiodic_field(geom, BC)), O.lookup_tables(geom)
    b = cnormal(rng, (nrhs, 4 if nd == 4 else 2, nc, vol))
    for herm in ([False] if nd == 3 else [False, True]):
        op = make_op(u, geom, kappa, herm, "fundamental")
        solver = dirac_solver.conjugate_gradient(tol=tol, precision="f64", delta=0.05, rhs_per_thread=1)
        x = solver.solve(op, cu(b))
        for i in range(nrhs):
            res = np.linalg.norm(b[i] - O.wilson_apply(ubc, x[i].cpu().numpy(), kappa, herm, tables))
            assert res < tol * np.linalg.norm(b[i]), (herm, i, solver.reports[i])
            assert solver.reports[i]["status"] == 0


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("values", [(1, 1, 1), (1, 1, 0.3), (1, 0.3, 0.3), (1, 0.99999, 0.9), (1, 0.5, 0.2),
                                    (1, 0.3, 0.23), (1, 0.5, 1e-2), (1, 1e-3, 1e-3), (1, 0.7, 1e-6)])
def test_projection_over_singular_values(cuda_device, nc, values):
    """Polar factors of matrices with given singular values (equal ones, the line between the
    two SU(3) forms, nearly singular ones), scales from 1e-6 to 1e6 and determinants of every
    phase. The factor is conditioned by the smallest singular value: about thirty roundings of
    1.1e-16 each, three times that times the condition number."""
    from tfleonardym_b200 import smearing
    rng = np.random.default_rng(nc)
    vol = 333
    u, v = (np.linalg.qr(cnormal(rng, (vol, nc, nc)))[0] for _ in range(2))
    s = np.array((values[0], values[2]) if nc == 2 else values)
    w = u @ v
    phase = np.exp(1j * (np.linspace(-0.99 * np.pi, 0.99 * np.pi, vol) - np.angle(np.linalg.det(w))) / nc)
    u *= phase[:, None, None]
    w *= phase[:, None, None]
    x = (u * s) @ v * 10.0 ** np.linspace(-6, 6, vol)[:, None, None]
    got = smearing.unitary_sqrt_projection(cu(np.transpose(x, (1, 2, 0))[None])).cpu().numpy()[0]
    det = np.linalg.det(w)
    want = np.transpose(w / np.exp(1j * np.angle(det) / nc)[:, None, None], (1, 2, 0))
    assert np.abs(got - want).max() < 1e-14 * max(values) / min(values)
    g = np.transpose(got, (2, 0, 1))
    assert np.abs(np.conj(np.swapaxes(g, 1, 2)) @ g - np.eye(nc)).max() < 1e-14


# threads of single vectors: 64152 and 72171 (between the waves of 56832 and 75776 threads), 131072
# (between the second and the third of them), 207360 (SU(2) takes pairs up to the third wave); an odd count
# stays with single vectors
@pytest.mark.parametrize("geom,nc,nvec", [((9, 9, 9, 11), 3, 8), ((9, 9, 9, 11), 2, 8), ((9, 9, 9, 11), 3, 9),
                                          ((8, 8, 8, 16), 3, 16), ((12, 12, 12, 12), 2, 10), ((12, 12, 12, 12), 3, 10)])
def test_operator_on_pairs_of_vectors(cuda_device, geom, nc, nvec):
    rng = np.random.default_rng(nvec + nc)
    vol = int(np.prod(geom))
    u = links(rng, geom, nc, unitary=False)
    ubc, tables = O.apply_time_bc(u, O.antiperiodic_field(geom, BC)), O.lookup_tables(geom)
    x = cnormal(rng, (nvec, 4, nc, vol))
    for herm in (False, True):
        op = make_op(u, geom, 0.12, herm, "fundamental")
        out = op.apply(cu(x)).cpu().numpy()
        for k in (0, nvec // 2, nvec - 1):
            assert relerr(out[k], O.wilson_apply(ubc, x[k], 0.12, herm, tables)) < TOL, (herm, k)
        for k in range(nvec):
            assert relerr(out[k], op.apply(cu(x[k])).cpu().numpy()) < TOL, (herm, k)
