"""GPU test of the straight-line quotients of the register-tiled energy kernels: the same bits of
silu and silu' as the kernel with plain divisions (taken by a network of another width), over a
dense sweep of pre-activations through the range where they are used and past its ends."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200.energy_rno import EnergyAnchors, EnergyDissipationRVERNO, RVERNOModelConfig  # noqa: E402

EQ, NEQ, EVO = ("equilibrium_energy.network.network", "nonequilibrium_energy.network.network", "state_evolution.network")


def _model(width: int) -> EnergyDissipationRVERNO:
    """One hidden layer that copies the strain, c = 0..5: the rates are silu of the strain and
    the stress its derivative, each multiplied by one and added to zeros (no anchors)."""
    w = {}
    for prefix, n_in, n_out in ((EQ, 6, 1), (NEQ, 12, 1), (EVO, 12, 6)):
        w[f"{prefix}.0.weight"], w[f"{prefix}.0.bias"] = torch.zeros(width, n_in), torch.zeros(width)
        w[f"{prefix}.2.weight"] = torch.zeros(n_out, width)
        if prefix != NEQ:
            for c in range(6):
                w[f"{prefix}.0.weight"][c, c] = 1.0
                w[f"{prefix}.2.weight"][c if prefix == EVO else 0, c] = 1.0
    w[f"{EVO}.2.bias"] = torch.zeros(6)
    model = EnergyDissipationRVERNO(RVERNOModelConfig("energy_rve_rno", "continuous", "cs_semi_implicit_forward_euler",
                                                      "direct_rate", 0.02, 6, width, 1, "silu"))  # fmt: skip
    model.load_state_dict(w)
    return model


def test_silu_and_its_derivative_have_the_bits_of_the_divisions() -> None:
    # every 499th float from 1e-30 to 120 of both signs (2^23 x 107 / 499 = 1.8 million each),
    # and 2^18 floats on either side of the range's end
    lo, hi = (int(np.float32(v).view(np.int32)) for v in (1.0e-30, 120.0))
    edge = int(np.float32(69.0).view(np.int32))
    bits = np.concatenate([np.arange(lo, hi, 499), np.arange(edge - 2**18, edge + 2**18)]).astype(np.int32)
    z = torch.as_tensor(bits.view(np.float32))
    z = torch.cat([z, -z, torch.zeros(12)])
    z = z[: z.numel() // 6 * 6].reshape(-1, 6)
    tiles, divisions = _model(128), _model(64)
    latent, step = torch.zeros(z.shape[0], 6), torch.zeros(z.shape[0])
    a, b = (m.update_batch(z, latent, step, EnergyAnchors(torch.zeros(14, device="cuda"))) for m in (tiles, divisions))
    assert torch.equal(a.dimensionless_state_rate, b.dimensionless_state_rate)
    assert torch.equal(a.stress, b.stress)
    assert bool((a.dimensionless_state_rate != 0).any()) and bool((a.stress != 0).any())
