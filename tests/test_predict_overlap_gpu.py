"""Latent states that lie in the buffers of a surrogate step: whole states are taken, a view
shifted by some points is refused (each point's next state would overwrite another's input)."""

from __future__ import annotations

import ctypes

import pytest
import torch

from concrete_impact_b200 import _native
from concrete_impact_b200.rno import RNOConfig, RNOSurrogate


def test_entry_point_refuses_shifted_latent_states_before_the_gpu() -> None:
    fake, points = 4096, 10
    w, x = _native.RNOWindowC(), _native.RNOPredictInputsC()
    w.B, w.T, w.hidden = points, 1, 128
    w.strain = w.rate = w.coef = w.err = fake
    w.z = 1 << 20
    for i in range(4):
        w.W[i], w.bias[i] = fake, fake
    x.strain = x.rate = x.stress = fake
    x.strain_scale = x.rate_scale = x.stress_scale = 1.0
    size = 4 * 6 * points  # bytes of a state
    for shift in (-size + 4, -24, 24, size - 4, size + 24, 2 * size - 4):
        x.z = (1 << 20) + shift
        assert _native.load_library().cib_rno_predict(ctypes.byref(w), ctypes.byref(x), None) == -1, shift


@pytest.mark.gpu
@pytest.mark.parametrize("points", [40, 7105, 37_888])
def test_predict_refuses_a_shifted_view_of_its_own_buffer(points: int) -> None:
    rno = RNOSurrogate(RNOConfig(seed=4))
    g = torch.Generator(device="cuda").manual_seed(points)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    strain, rate, z, coef = r(points, 6), r(points, 6), r(points, 6), 0.05 * torch.rand(points, generator=g, device="cuda")
    buffers = rno.predict(strain, rate, z, coef)[2]
    flat = buffers["z"].view(-1, 6)
    with pytest.raises(RuntimeError):  # as torch refuses to copy between overlapping tensors
        rno.predict(strain, rate, flat[3 : 3 + points], coef, buffers)
    for start in (0, points):  # the state that went in, the state that came out
        want = flat[start : start + points].clone()
        expected = rno.predict(strain, rate, want, coef)
        got = rno.predict(strain, rate, flat[start : start + points], coef, buffers)
        assert torch.equal(got[0], expected[0]) and torch.equal(got[1], expected[1])
        assert torch.equal(buffers["z"][0], want)


@pytest.mark.gpu
def test_strain_in_the_step_s_own_buffer_is_read_before_it_is_written() -> None:
    points, rno = 37_888, RNOSurrogate(RNOConfig(seed=4))
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    rate, z, coef = r(points, 6), r(points, 6), 0.05 * torch.rand(points, generator=g, device="cuda")
    buffers = rno.predict(r(points, 6), rate, z, coef)[2]
    strain = buffers["z"].view(-1, 6)[3 : 3 + points]
    expected = rno.predict(strain.clone(), rate, z, coef)
    got = rno.predict(strain, rate, z, coef, buffers)
    assert torch.equal(got[0], expected[0]) and torch.equal(got[1], expected[1])
