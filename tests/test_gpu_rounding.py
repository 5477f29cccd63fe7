"""Rounding of the gauge and force kernels against extended precision (80-bit, so that the
reference's own rounding, which is the kernels' in 64 bits, does not count).

Bounds, relative in the 2-norm: what the plainest evaluation gives -- every product formed by itself,
then added -- and 5 % for the draw of the inputs.  Products that accumulate into a long sum lie 20 to
35 % above, short-cut angles 6 %.
"""
import numpy as np
import pytest
import torch

from oracle import lym_oracle as O
from tests.test_gpu_kernel_edges import cnormal, cu, smooth_links

pytestmark = pytest.mark.gpu

L, CL = np.longdouble, np.clongdouble


def mm(a, b):
    return np.einsum("ijv,jkv->ikv", a, b)


def dag(a):
    return np.conj(np.swapaxes(a, 0, 1))


def off(got, exact):
    got = got.cpu().numpy() if isinstance(got, torch.Tensor) else got
    return float(np.sqrt(np.sum(np.abs(got - exact) ** 2) / np.sum(np.abs(exact) ** 2)))


def momenta(rng, geom, nc):
    x = 0.5 * cnormal(rng, (len(geom), nc, nc, int(np.prod(geom))))
    p = x - np.conj(np.swapaxes(x, 1, 2))
    return p - np.einsum("miiv->mv", p)[:, None, None] * (np.eye(nc) / nc)[None, :, :, None]


def configuration(u, geom):
    from tfleonardym_b200 import lattice as lt
    return lt.Configuration(cu(u), geom, u.shape[1], len(geom))


# plainest: 1.14e-16 and 1.35e-16
@pytest.mark.parametrize("nc,bound", [(2, 1.2e-16), (3, 1.42e-16)])
def test_gauge_force(cuda_device, nc, bound):
    from tfleonardym_b200 import gauge_action, staples
    geom, beta = (6, 6, 6, 8), 5.5
    rng = np.random.default_rng(nc)
    u, tables = smooth_links(rng, geom, nc, spread=0.25), O.lookup_tables(geom)
    x = u.astype(CL)
    exact, sums = [], []
    for mu in range(4):
        s = np.zeros(x.shape[1:], CL)
        for nu in range(4):
            if nu != mu:
                s += mm(mm(x[nu], O.translate(x[mu], tables, nu, 1)), dag(O.translate(x[nu], tables, mu, 1)))
                s += O.translate(mm(mm(dag(x[nu]), x[mu]), O.translate(x[nu], tables, mu, 1)), tables, nu, -1)
        w = mm(x[mu], dag(s))
        f = -L(beta) / (4 * nc) * (dag(w) - w)
        sums.append(s)
        exact.append(f - np.einsum("iiv->v", f) / nc * np.eye(nc)[:, :, None])
    action = gauge_action.yang_mills(configuration(u, geom), beta)
    assert off(action.force(), np.stack(exact)) < bound
    assert off(staples.get_staple_sums(action.cfg, -1), np.stack(sums)) < bound
    p = momenta(rng, geom, nc)
    kicked = action.kicked_momenta(cu(p), 1.0).cpu().numpy()
    assert off(kicked, p.astype(CL) + np.stack(exact)) < bound
    assert np.array_equal(action.kick_and_drift(cu(p), 1.0, 0.1)[0].cpu().numpy(), kicked)


# plainest: 1.87e-16 in 4D
@pytest.mark.parametrize("geom", [(4, 4, 6, 6), (16, 24)])
@pytest.mark.parametrize("nc", [2, 3])
def test_fundamental_force_of_several_poles(cuda_device, nc, geom):
    from tfleonardym_b200 import boundary_conditions as bc
    from tfleonardym_b200 import dirac
    rng = np.random.default_rng(10 * nc + len(geom))
    nd, vol, kappa, alphas = len(geom), int(np.prod(geom)), 0.12, [0.7, -1.3, 0.2, 0.9]
    u, tables = smooth_links(rng, geom, nc, spread=0.25), O.lookup_tables(geom)
    x, y = (cnormal(rng, (4, 4 if nd == 4 else 2, nc, vol)) for _ in range(2))
    g, gd = (m.astype(CL) for m in O.gammas(nd))
    one = np.eye(g.shape[1]).astype(CL)
    last = np.arange(vol) % geom[-1] == geom[-1] - 1
    exact = []
    for mu in range(nd):
        sign = np.where(last, -1, 1) if mu == nd - 1 else np.ones(vol, int)
        f = np.zeros((nc, nc, vol), CL)
        for w, a, b in zip(alphas, x.astype(CL), y.astype(CL)):
            for p, q in ((a, b), (b, a)):
                z = np.einsum("ijv,njv->niv", u[mu].astype(CL), O.translate(q, tables, mu, 1)) * sign
                d = np.einsum("miv,mn,njv->jiv", np.conj(p), gd @ (one - g[mu]), z)
                d -= np.einsum("miv,mn,njv->jiv", np.conj(z), gd @ (one + g[mu]), p)
                f += L(w) * L(kappa) / 2 * (d - np.einsum("iiv->v", d) / nc * np.eye(nc)[:, :, None])
        exact.append(f)
    op = dirac.DiracWilsonOperator(configuration(u, geom), kappa, True, representation="fundamental",
                                   boundary_condition_provider=bc.time_antiperiodic_provider(-1))
    force = op.accumulate_force(torch.zeros_like(op.cfg.gauge_field), alphas, cu(x), cu(y), symmetric=True)
    assert off(force, np.stack(exact)) < 1.96e-16


# plainest: 1.47e-16
@pytest.mark.parametrize("eps", [0.01, 0.1])
def test_drift(cuda_device, eps):
    from tfleonardym_b200 import hmc
    geom, nc = (6, 6, 6, 8), 3
    rng = np.random.default_rng(5)
    u, p = smooth_links(rng, geom, nc, spread=0.25), momenta(rng, geom, nc)
    exact = []
    for mu in range(4):
        x = p[mu].astype(CL) * L(eps)
        term = total = np.broadcast_to(np.eye(nc, dtype=CL)[:, :, None], x.shape)
        for k in range(1, 40):
            term = mm(term, x) / k
            total = total + term
        exact.append(mm(total, u[mu].astype(CL)))
    assert off(hmc.update_link_field(cu(u), cu(p), eps), np.stack(exact)) < 1.54e-16


# plainest: 1.08e-16
def test_traces_of_four_links(cuda_device):
    from tfleonardym_b200 import _dev, _lib, measurements
    geom, nc, bound = (6, 6, 6, 8), 3, 1.13e-16
    rng = np.random.default_rng(nc)
    u, tables = smooth_links(rng, geom, nc, spread=0.25), O.lookup_tables(geom)
    x, cfg = u.astype(CL), configuration(u, geom)
    total = 0
    for a in range(4):
        for b in range(a + 1, 4):
            loop = mm(mm(x[a], O.translate(x[b], tables, a, 1)), dag(mm(x[b], O.translate(x[a], tables, b, 1))))
            trace = np.einsum("iiv->v", loop)
            assert off(measurements.path_field(cfg, [a + 1, b + 1, -a - 1, -b - 1]), trace) < bound, (a, b)
            total = total + trace
    plaquettes, squares = (torch.empty(u.shape[-1], dtype=torch.complex128, device="cuda") for _ in range(2))
    _lib.check(_lib.lib().lym_plane_loops(measurements._lattice(cfg).handle, nc, _dev.ptr(cfg.gauge_field), -1,
                                          _dev.ptr(plaquettes), _dev.ptr(squares), _dev.stream()), "lym_plane_loops")
    assert off(plaquettes, total) < bound
