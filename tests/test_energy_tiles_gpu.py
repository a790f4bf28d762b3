"""GPU tests of the register-tiled energy RVE-RNO kernels (hidden width 128): update and
algorithmic tangent against a float64 evaluation of the same FP32 weights with autograd, at the
edges of the tiles and of the rules that choose them, and the branch for pre-activations beyond
the range of the straight-line quotients."""

from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200.energy_rno import EnergyDissipationRVERNO, RVERNOModelConfig  # noqa: E402

EQ, NEQ, EVO = ("equilibrium_energy.network.network", "nonequilibrium_energy.network.network", "state_evolution.network")
ULP = 2.0**-24  # of an FP32 rounding


def _weights(layers: int, latent: int, seed: int) -> dict[str, torch.Tensor]:
    g, out = torch.Generator().manual_seed(seed), {}
    for prefix, n_in, n_out in ((EQ, 6, 1), (NEQ, 6 + latent, 1), (EVO, 6 + latent, latent)):
        for layer in range(layers + 1):
            fan, rows = (n_in if layer == 0 else 128), (128 if layer < layers else n_out)
            out[f"{prefix}.{2 * layer}.weight"] = (3.0 * torch.rand(rows, fan, generator=g) - 1.5) / math.sqrt(fan)
            if layer < layers or prefix == EVO:
                out[f"{prefix}.{2 * layer}.bias"] = (torch.rand(rows, generator=g) - 0.5) / math.sqrt(fan)
    return out


def _model(layers: int, latent: int, integrator: str, weights) -> EnergyDissipationRVERNO:
    model = EnergyDissipationRVERNO(RVERNOModelConfig("energy_rve_rno", "continuous", integrator, "direct_rate", 0.02,
                                                      latent, 128, layers, "silu"))  # fmt: skip
    model.load_state_dict(weights)
    return model


def _reference(weights, layers: int, integrator: str, strain, latent, step, tangent: bool) -> dict:
    w = {k: v.double() for k, v in weights.items()}

    def net(prefix, x):
        for layer in range(layers):
            x = torch.nn.functional.silu(x @ w[f"{prefix}.{2 * layer}.weight"].T + w[f"{prefix}.{2 * layer}.bias"])
        y = x @ w[f"{prefix}.{2 * layers}.weight"].T
        return y + w[f"{prefix}.{2 * layers}.bias"] if prefix == EVO else y

    def gradient(prefix, x):
        return torch.autograd.grad(net(prefix, x).sum(), x, create_graph=True)[0]

    e = strain.double().requires_grad_(True)
    z = latent.double()
    zero = torch.zeros(1, 6 + z.shape[1], dtype=torch.float64, requires_grad=True)
    rate = net(EVO, torch.cat([e, z], 1))
    after = z + step.double()[:, None] / 0.02 * rate
    at = after if integrator == "current_state_stress_forward_euler" else z
    stress = gradient(EQ, e) - gradient(EQ, zero[:, :6]) + (gradient(NEQ, torch.cat([e, at], 1)) - gradient(NEQ, zero))[:, :6]
    out = {"stress": stress.detach(), "latent_state": after.detach(), "dimensionless_state_rate": rate.detach()}
    if tangent:
        rows = [torch.autograd.grad(stress[:, i].sum(), e, retain_graph=True)[0] for i in range(6)]
        out["tangent"] = torch.stack(rows, 1)
    return out


# Points: one; one past a 16-point tile; one past the 8-point tiles' reach (1185), the 16-point
# tiles' (4737) on 148 SMs; several waves.  Tolerance of a field's 2-norm: a result passes
# through at most 3 (L + 1) sums of up to 128 terms (state, gradient, direction) plus as many
# activations, one rounding per term: 3 (L + 1) (128 + 8) 2^-24 to first order.
@pytest.mark.parametrize("points, layers, latent, integrator, tangent", [
    (1, 4, 6, "current_state_stress_forward_euler", True),
    (17, 4, 6, "cs_semi_implicit_forward_euler", True),
    (1185, 4, 6, "current_state_stress_forward_euler", True),
    (40, 3, 8, "current_state_stress_forward_euler", True),
    (9, 2, 1, "current_state_stress_forward_euler", True),
    (33, 1, 3, "cs_semi_implicit_forward_euler", False),
    (4737, 4, 6, "current_state_stress_forward_euler", False),
    (20011, 2, 6, "current_state_stress_forward_euler", False),
])  # fmt: skip
def test_tiles_match_a_float64_evaluation(points, layers, latent, integrator, tangent) -> None:
    weights = _weights(layers, latent, seed=points)
    model = _model(layers, latent, integrator, weights)
    g = torch.Generator().manual_seed(points + 1)
    strain, state = torch.randn(points, 6, generator=g), torch.randn(points, latent, generator=g)
    step = 0.02 * torch.rand(points, generator=g)
    ref = _reference(weights, layers, integrator, strain, state, step, tangent)
    got = model.update_batch(strain, state, step, model.prepare_energy_anchors(), compute_tangent=tangent)
    tol = 3 * (layers + 1) * (128 + 8) * ULP
    for name, exact in ref.items():
        error = (getattr(got, name).double().cpu() - exact).norm() / exact.norm()
        assert error <= tol, (name, float(error), tol)


def test_pre_activations_beyond_the_straight_line_range() -> None:
    """One hidden layer whose pre-activations are its biases, exactly, out to where 1 + e^-z
    overflows: the rates are sums of 129 exact products' roundings, and no stress arises."""
    weights = _weights(1, 6, seed=3)
    bias = torch.linspace(-300.0, 300.0, 128)
    bias[::9] = torch.tensor([69.0, -69.0, 69.5, -69.5, -87.5, -88.5, 88.5, -104.0, 0.0, -1e-30, 1e30, -1e30, -17.0, 17.0,
                              1e-38])  # fmt: skip
    for prefix in (EQ, NEQ, EVO):
        weights[f"{prefix}.0.weight"].zero_()
        weights[f"{prefix}.0.bias"] = bias.clone()
    model = _model(1, 6, "current_state_stress_forward_euler", weights)
    got = model.update_batch(torch.ones(5, 6), torch.ones(5, 6), torch.ones(5), model.prepare_energy_anchors())
    h = torch.nn.functional.silu(bias.double())
    terms = weights[f"{EVO}.2.weight"].double() * h
    exact = terms.sum(1) + weights[f"{EVO}.2.bias"].double()
    bound = (129 + 8) * ULP * (terms.abs().sum(1) + weights[f"{EVO}.2.bias"].double().abs())
    assert ((got.dimensionless_state_rate.double().cpu() - exact).abs() <= bound).all()
    assert (got.stress == 0).all()
