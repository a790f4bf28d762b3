"""GPU tests of PhasedMaterialModel around materials written with torch: derivatives pass through
its gather and scatter (backward and forward mode), and arrays that a raw copy cannot take are
placed or refused as torch's index_copy_ does."""

from __future__ import annotations

import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as fwd

pytestmark = pytest.mark.gpu

from concrete_impact_b200.materials import (DEFAULT_RESPONSE_REQUIREMENTS, J2ViscoplasticMaterial,  # noqa: E402
                                            MaterialPointRequest, MaterialPointResponse, MaterialResponseRequirements,
                                            MaterialState, MaterialUpdateSettings, PhasedMaterialModel, RVEPhase)  # fmt: skip

IDS = np.array([0, 1, 1, 0, 0, 1, 0] * 5)


class Cubic:
    """Stress 3 e^2 + rate, energy sum e^3; every array passes through ``form`` on its way out."""

    name, density, maximum_wave_speed = "cubic", 1.0, 1.0

    def __init__(self, form=lambda t: t) -> None:
        self.form = form

    def initialize_state(self, n_points: int) -> MaterialState:
        return MaterialState({})

    def update(self, request, state, requirements=DEFAULT_RESPONSE_REQUIREMENTS) -> MaterialPointResponse:
        e = request.strains
        return MaterialPointResponse(self.form(3.0 * e**2 + request.strain_rates), state, free_energy=self.form((e**3).sum(1)),
                                     diagnostics={"norm": self.form((e**2).sum(1)), "count": torch.ones_like(e[:, 0])})  # fmt: skip


def _update(eps, rate, form=lambda t: t):
    j2 = J2ViscoplasticMaterial("mortar", 2200.0, 25.0e9, 0.2, 20.0e6, 2.0e9, 1.0e-3, 20.0e6, 1.0)
    model = PhasedMaterialModel("rve", (RVEPhase("c", Cubic(form)), RVEPhase("j", j2)), IDS, 2400.0)
    request = MaterialPointRequest(eps, rate, 1e-4, "three_dimensional", MaterialUpdateSettings(50, 1.0e-10, 1.0e-12, 1.0e-10))
    return model.update(request, model.initialize_state(IDS.size), MaterialResponseRequirements(False, True, False))


def _inputs():
    g = torch.Generator(device="cuda").manual_seed(2)
    eps = 1e-3 * torch.randn((IDS.size, 6), generator=g, device="cuda", dtype=torch.float64)
    return eps, torch.randn((IDS.size, 6), generator=g, device="cuda", dtype=torch.float64)


def test_backward_reaches_the_strains_of_a_torch_material() -> None:
    eps, rate = _inputs()
    plain = _update(eps, rate)
    eps.requires_grad_(True)
    rate.requires_grad_(True)
    out = _update(eps, rate)
    cubic = torch.as_tensor(IDS == 0, device="cuda")[:, None]
    assert torch.equal(out.stresses.detach(), plain.stresses) and torch.equal(out.free_energy.detach(), plain.free_energy)
    for name, values in plain.diagnostics.items():
        torch.testing.assert_close(out.diagnostics[name].detach(), values, rtol=0.0, atol=0.0, equal_nan=True)
    assert not out.diagnostics["count"].requires_grad
    grads = torch.autograd.grad(out.stresses.sum(), (eps, rate), retain_graph=True)
    torch.testing.assert_close(grads[0], torch.where(cubic, 6.0 * eps, 0.0 * eps))
    torch.testing.assert_close(grads[1], torch.where(cubic, 1.0, 0.0 * eps))
    norm = out.diagnostics["norm"][cubic[:, 0]].sum()
    grad = torch.autograd.grad(out.free_energy.sum() + norm, eps)[0]
    torch.testing.assert_close(grad, torch.where(cubic, 3.0 * eps**2 + 2.0 * eps, 0.0 * eps))


def test_forward_mode_reaches_the_stress_of_a_torch_material() -> None:
    eps, rate = _inputs()
    direction = torch.randn_like(eps)
    with fwd.dual_level():
        out = _update(fwd.make_dual(eps, direction), rate)
        tangent = fwd.unpack_dual(out.stresses).tangent
    cubic = torch.as_tensor(IDS == 0, device="cuda")[:, None]
    torch.testing.assert_close(tangent, torch.where(cubic, 6.0 * eps * direction, 0.0 * eps))


def test_arrays_that_are_not_plain_device_doubles() -> None:
    eps, rate = _inputs()
    plain = _update(eps, rate)
    strided = _update(eps, rate, lambda t: torch.stack([t, t], -1)[..., 0])
    assert torch.equal(strided.stresses, plain.stresses) and torch.equal(strided.free_energy, plain.free_energy)
    for form in (lambda t: t.float(), lambda t: t.cpu(), lambda t: t[:-1]):
        with pytest.raises((RuntimeError, IndexError)):
            _update(eps, rate, form)
