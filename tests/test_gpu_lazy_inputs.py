"""Tensors whose values differ from their memory: torch keeps a conjugate or a sign as a flag of
the tensor, and the kernels read memory.  Every entry point has to give what it gives for the same
values written out, bit for bit (the same kernel on the same numbers).
"""
import numpy as np
import pytest
import torch

from oracle import lym_oracle as O
from tests.conftest import relerr
from tests.test_gpu_kernel_edges import cnormal, cu, links, make_op, smooth_links

pytestmark = pytest.mark.gpu


def conj_flagged(t):
    x = t.conj().resolve_conj().conj()
    assert x.is_conj() and torch.equal(x.resolve_conj(), t)
    return x


def sign_flagged(t):
    x = torch._neg_view(-t)
    assert x.is_neg() and torch.equal(x.resolve_neg(), t)
    return x


def both_flagged(t):
    x = torch._neg_view(conj_flagged(-t))
    assert x.is_conj() and x.is_neg() and torch.equal(x.resolve_conj().resolve_neg(), t)
    return x


FORMS = [conj_flagged, sign_flagged, both_flagged]


def momenta(rng, geom, nc):
    x = cnormal(rng, (len(geom), nc, nc, int(np.prod(geom))))
    p = 0.5 * (x - np.conj(np.swapaxes(x, 1, 2)))
    return p - np.einsum("miiv->mv", p)[:, None, None] * (np.eye(nc) / nc)[None, :, :, None]


@pytest.mark.parametrize("form", FORMS)
def test_molecular_dynamics_of_flagged_tensors(cuda_device, form):
    from tfleonardym_b200 import gauge_action, hmc
    from tfleonardym_b200 import lattice as lt
    rng = np.random.default_rng(8)
    geom, nc = (4, 3, 2, 5), 3
    u, p, f = cu(smooth_links(rng, geom, nc)), cu(momenta(rng, geom, nc)), cu(momenta(rng, geom, nc))
    assert relerr(hmc.update_momenta(form(p), f, 0.3).cpu(), O.update_momenta(p.cpu().numpy(), f.cpu().numpy(), 0.3)) < 1e-13
    assert torch.equal(hmc.update_momenta(form(p), form(f), 0.3), hmc.update_momenta(p, f, 0.3))
    assert torch.equal(hmc.update_link_field(form(u), form(p), 0.1), hmc.update_link_field(u, p, 0.1))

    def configuration(t):
        return lt.Configuration(t, geom, nc, len(geom))

    plain = gauge_action.yang_mills(configuration(u), 5.5)
    flagged = gauge_action.yang_mills(configuration(form(u)), 5.5)
    assert torch.equal(flagged.force(), plain.force()) and flagged.energy() == plain.energy()
    assert torch.equal(flagged.kicked_momenta(form(p), 0.2), plain.kicked_momenta(p, 0.2))
    for a, b in zip(flagged.kick_and_drift(form(p), 0.2, 0.1), plain.kick_and_drift(p, 0.2, 0.1)):
        assert torch.equal(a, b)
    assert hmc.momenta_energy(form(p)) == hmc.momenta_energy(p)
    for integrate in (hmc.integrate_om, hmc.integrate_lp):
        c0, p0 = integrate(configuration(u), p, [plain], [2], 0.1)
        c1, p1 = integrate(configuration(form(u)), form(p), [flagged], [2], 0.1)
        assert torch.equal(c0.gauge_field, c1.gauge_field) and torch.equal(p0, p1)
    # in place on the caller's tensors
    cs = [configuration(u.clone()), configuration(form(u))]
    ps = [p.clone(), form(p)]
    hmc.gauge_step_lattices(cs, ps, [5.5, 5.5], 0.2, 0.1)
    assert not torch.equal(ps[0], p)
    assert torch.equal(ps[1].resolve_conj().resolve_neg(), ps[0])
    assert torch.equal(cs[1].gauge_field.resolve_conj().resolve_neg(), cs[0].gauge_field)


@pytest.mark.parametrize("form", FORMS)
def test_operators_and_observables_of_flagged_tensors(cuda_device, form):
    from tfleonardym_b200 import _dev, dirac_solver, gauge_action, measurements, smearing, staples
    from tfleonardym_b200 import lattice as lt
    rng = np.random.default_rng(9)
    geom, nc = (4, 2, 4, 6), 3
    vol = int(np.prod(geom))
    u = links(rng, geom, nc)
    plain, flagged = (lt.Configuration(t, geom, nc, 4) for t in (cu(u), form(cu(u))))
    for call in (lambda c: staples.get_staple_sums(c), lambda c: smearing.ape_smearing(c, 0.3).gauge_field,
                 lambda c: smearing.unitary_sqrt_projection(c.gauge_field),
                 lambda c: measurements.path_field(c, [1, 2, -1, -2])):
        assert torch.equal(call(flagged), call(plain))
    assert gauge_action.plaquette_trace_sum(flagged) == gauge_action.plaquette_trace_sum(plain)
    for a, b in zip(measurements.glueball_operators(flagged) + measurements.polyakov_operators(flagged),
                    measurements.glueball_operators(plain) + measurements.polyakov_operators(plain)):
        assert np.array_equal(a.value, b.value)
    for representation, shape in (("fundamental", (2, 4, nc, vol)), ("adjoint", (2, 4, nc, nc, vol))):
        op = make_op(u, geom, 0.11, True, representation)
        x, y = cu(cnormal(rng, shape)), cu(cnormal(rng, shape))
        assert torch.equal(op.apply(form(x)), op.apply(x))
        zero = torch.zeros_like(op.cfg.gauge_field)
        assert torch.equal(op.accumulate_force(zero.clone(), [0.7, -0.4], form(x), form(y)),
                           op.accumulate_force(zero.clone(), [0.7, -0.4], x, y))
    b = cu(cnormal(rng, (4, nc, vol)))
    assert _dev.cdot(form(b), b) == _dev.cdot(b, b)
    assert torch.equal(_dev.axpby(0.5, form(b), 2.0, form(b)), _dev.axpby(0.5, b, 2.0, b))
    op = make_op(u, geom, 0.11, False, "fundamental")
    for rhs_per_thread in (0, 1):
        solver = dirac_solver.conjugate_gradient(tol=1e-10, rhs_per_thread=rhs_per_thread)
        assert torch.equal(solver.solve(op, form(b)), solver.solve(op, b))


@pytest.mark.parametrize("geom,nc", [((5, 7), 2), ((3, 5, 2), 3), ((4, 3, 2, 5), 3), ((4, 3, 2, 5), 2)])
def test_updates_in_place(cuda_device, geom, nc):
    """The entry points a host calls on its own fields, and those whose output may be their input:
    the bits of the call into another buffer."""
    from tfleonardym_b200 import _dev, _lib, gauge_action, hmc
    from tfleonardym_b200 import lattice as lt
    rng = np.random.default_rng(int(np.prod(geom)))
    nd, vol, L = len(geom), int(np.prod(geom)), _lib.lib()
    u, p, f = cu(smooth_links(rng, geom, nc)), cu(momenta(rng, geom, nc)), cu(momenta(rng, geom, nc))
    lat, st = lt.get_lattice(geom).handle, _dev.stream()
    for reunitarize in (0, 1):
        want = hmc.update_link_field(u, p, 0.1, reunitarize=bool(reunitarize))
        for entry in ("update", "drift"):
            x = u.clone()
            if entry == "update":
                rc = L.lym_update_links(nd, nc, vol, _dev.ptr(x), _dev.ptr(p), 0.1, reunitarize, st)
            else:
                rc = L.lym_link_drift(nd, nc, vol, _dev.ptr(x), _dev.ptr(p), 0.1, reunitarize, _dev.ptr(x), st)
            assert rc == 0 and torch.equal(x, want), (entry, reunitarize)
    want = hmc.update_momenta(p, f, 0.3)
    for entry in ("update", "kick"):
        x = p.clone()
        if entry == "update":
            rc = L.lym_update_momenta(p.numel(), _dev.ptr(x), _dev.ptr(f), 0.3, st)
        else:
            rc = L.lym_momenta_kick(p.numel(), _dev.ptr(x), _dev.ptr(f), 0.3, _dev.ptr(x), st)
        assert rc == 0 and torch.equal(x, want), entry
    action = gauge_action.yang_mills(lt.Configuration(u, geom, nc, nd), 5.5)
    want = action.kicked_momenta(p, 0.2)
    x = p.clone()
    assert action.force_into_momenta(x, 0.2) is x and torch.equal(x, want)
    x = p.clone()
    assert L.lym_gauge_kick(lat, nc, 5.5, _dev.ptr(u), _dev.ptr(x), 0.2, _dev.ptr(x), st) == 0
    assert torch.equal(x, want)
    p_want, u_want = action.kick_and_drift(p, 0.2, 0.1)
    x, y = p.clone(), torch.empty_like(u)
    assert L.lym_gauge_kick_drift(lat, nc, 5.5, _dev.ptr(u), _dev.ptr(x), 0.2, 0.1, _dev.ptr(x), _dev.ptr(y), st) == 0
    assert torch.equal(x, p_want) and torch.equal(y, u_want)
