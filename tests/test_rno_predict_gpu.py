"""GPU test of one inference step from physical inputs: the same bits as normalising with torch
(a division by a number is a product with its reciprocal), stepping on the normalised inputs and
scaling the stress, for every input type, in each kernel's range of points."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200.rno import RNOConfig, RNOScales, RNOSurrogate  # noqa: E402

F32, F64 = torch.float32, torch.float64


# points: the narrow kernel (7,104 is its last on 148 SMs), the window kernel, the inference kernel
@pytest.mark.parametrize("points", [1, 17, 7104, 7105, 37_760, 37_888])
@pytest.mark.parametrize("strain_type, rate_type, layout", [(F64, F64, "plain"), (F32, F32, "plain"), (F64, F32, "plain"),
                                                            (F32, F64, "strided"), (F64, F64, "own latent")])  # fmt: skip
def test_predict_equals_torch_around_the_normalised_step(points, strain_type, rate_type, layout) -> None:
    g = torch.Generator(device="cuda").manual_seed(points)
    scales = RNOScales(1.3e-3, 7.7, 2.1e7)
    rno = RNOSurrogate(RNOConfig(seed=4), scales)
    rno.set_elastic_skip((2.0e10 * (torch.eye(6) + 0.1)).numpy())
    field = lambda scale, kind: (scale * torch.randn((points, 6), generator=g, device="cuda", dtype=F64)).to(kind)  # noqa: E731
    strain, rate, z = field(1e-3, strain_type), field(8.0, rate_type), field(0.5, F32)
    coef = torch.rand(points, generator=g, device="cuda") * 0.05
    both, stress_n = torch.empty((2, points, 6), device="cuda"), torch.empty((points, 6), device="cuda")
    both[0] = z
    rno.predict_normalized((strain / scales.strain).float(), (rate / scales.rate).float(), coef, both, stress_n)
    buffers = None
    if layout == "strided":
        strain = torch.cat([strain, strain], 1)[:, :6]
    elif layout == "own latent":  # the latent state that a step returned
        buffers = rno.predict(strain, rate, z, coef)[2]
        buffers["z"][1] = z
        z = buffers["z"][1]
    stress, latent, buffers = rno.predict(strain, rate, z, coef, buffers)
    assert torch.equal(stress, stress_n * scales.stress) and torch.equal(latent, both[1])
    assert torch.equal(buffers["z"][0], both[0]) and torch.equal(buffers["stress"][0], stress_n)
