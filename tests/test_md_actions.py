"""Actions a user gives the integrators: what the object itself says about its kick and its links
counts, also where it is a plain gauge action otherwise.  The device calls are stood in for."""
import types

import pytest
import torch

from tfleonardym_b200 import gauge_action, hmc
from tfleonardym_b200 import lattice as lt


@pytest.fixture
def device_calls(monkeypatch):
    """Kernels of the gauge action and the drift, in numbers: a kick adds w, a drift adds w P."""
    calls = []

    def kicked(self, momenta, w):
        calls.append("kick")
        return momenta + w

    def kick_and_drift(self, momenta, w, e):
        calls.append("both")
        return momenta + w, self.cfg.gauge_field + e * (momenta + w)

    def update(config, momenta, w):
        calls.append("drift")
        return lt.Configuration(config.gauge_field + w * momenta, config.geometry, config.colors,
                                config.number_of_dimensions)

    monkeypatch.setattr(gauge_action.yang_mills, "kicked_momenta", kicked)
    monkeypatch.setattr(gauge_action.yang_mills, "kick_and_drift", kick_and_drift)
    monkeypatch.setattr(hmc, "update_configuration", update)
    return calls


def start():
    cfg = lt.Configuration(torch.ones(3, dtype=torch.complex128), (2, 2), 2, 2)
    return cfg, torch.full((3,), 0.5, dtype=torch.complex128)


def reference(p, u, ops, kick):
    for op in ops:
        if op.kind == hmc.DRIFT:
            u = u + op.weight * p
        else:
            p = kick(p, op.weight)
    return u, p


def test_the_plain_gauge_action_takes_the_fused_kernels(device_calls):
    cfg, p = start()
    ops = hmc.schedule("omelyan", [2], 0.1)
    c1, p1 = hmc.run_schedule(cfg, p, [gauge_action.yang_mills(cfg, 5.5)], ops)
    u, q = reference(p, cfg.gauge_field, ops, lambda p, w: p + w)
    assert "both" in device_calls
    assert torch.allclose(p1, q) and torch.allclose(c1.gauge_field, u)


@pytest.mark.parametrize("given_to", ["object", "class"])
def test_an_own_force_into_momenta_is_called(device_calls, monkeypatch, given_to):
    cfg, p = start()
    action = gauge_action.yang_mills(cfg, 5.5)

    def own(self, momenta, w):
        return momenta.mul_(1 + w)

    if given_to == "object":
        action.force_into_momenta = types.MethodType(own, action)
    else:
        monkeypatch.setattr(gauge_action.yang_mills, "force_into_momenta", own)
    ops = hmc.schedule("omelyan", [2], 0.1)
    c1, p1 = hmc.run_schedule(cfg, p, [action], ops)
    u, q = reference(p, cfg.gauge_field, ops, lambda p, w: p * (1 + w))
    assert set(device_calls) == {"drift"}
    assert torch.allclose(p1, q) and torch.allclose(c1.gauge_field, u)


def test_an_action_on_other_links_leaves_the_drift_to_the_configuration(device_calls):
    cfg, p = start()
    action = gauge_action.yang_mills(cfg, 5.5)

    def set_fat(config):  # an action that sees fat links
        action.cfg = lt.Configuration(2 * config.gauge_field, config.geometry, config.colors,
                                      config.number_of_dimensions)

    action.set_gauge_configuration = set_fat
    ops = hmc.schedule("omelyan", [2], 0.1)
    c1, p1 = hmc.run_schedule(cfg, p, [action], ops)
    u, q = reference(p, cfg.gauge_field, ops, lambda p, w: p + w)
    assert "both" not in device_calls
    assert torch.allclose(p1, q) and torch.allclose(c1.gauge_field, u)
