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
