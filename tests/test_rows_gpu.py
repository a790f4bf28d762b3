"""GPU tests of the row gather and scatter of a phased material (cib_copy_rows): exact copies."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import _native  # noqa: E402
from concrete_impact_b200.materials import (J2ViscoplasticMaterial, LinearElasticMaterial, MaterialPointRequest,  # noqa: E402
                                            MaterialResponseRequirements, MaterialState, MaterialUpdateSettings,
                                            PhasedMaterialModel, RVEPhase)  # fmt: skip


@pytest.mark.parametrize("count", [0, 1, 255, 256, 257, 70001])
def test_gather_and_scatter_of_several_widths(count: int) -> None:
    g = torch.Generator(device="cuda").manual_seed(count)
    n = 2 * count + 3
    ids = torch.randperm(n, generator=g, device="cuda")[:count]
    widths = [1, 6, 36] + [1] * 31  # more arrays than one launch takes
    new = lambda rows, w: torch.randn((rows, w), generator=g, device="cuda", dtype=torch.float64)  # noqa: E731
    far, near = [new(n, w) for w in widths], [new(count, w) for w in widths]
    got = [torch.empty_like(a) for a in near]
    _native.copy_rows(ids, [(a, to, w, 0.0) for a, to, w in zip(far, got, widths)], scatter=False)
    assert all(torch.equal(to, a[ids]) for a, to in zip(far, got))
    expected = [a.clone().index_copy_(0, ids, b) for a, b in zip(far, near)]
    expected[3][ids] = float("nan")
    _native.copy_rows(ids, [(None if i == 3 else b, a, w, float("nan")) for i, (a, b, w) in enumerate(zip(far, near, widths))],
                      scatter=True)  # fmt: skip
    for a, b in zip(far, expected):
        torch.testing.assert_close(a, b, rtol=0.0, atol=0.0, equal_nan=True)


@pytest.mark.parametrize("stray", [False, True])
def test_phased_update_places_every_phase(stray: bool) -> None:
    """Each phase's points as its material alone gives them; points of no phase are zero, and
    diagnostics that a phase lacks are NaN."""
    ids = np.array([0, 1, 1, 0, 0, 1, 0] * 40)
    if stray:
        ids[::11] = 9
    j2 = J2ViscoplasticMaterial("mortar", 2200.0, 25.0e9, 0.2, 20.0e6, 2.0e9, 1.0e-3, 20.0e6, 1.0)
    elastic = LinearElasticMaterial("aggregate", 2600.0, 50.0e9, 0.2)
    model = PhasedMaterialModel("rve", (RVEPhase("j", j2), RVEPhase("e", elastic), RVEPhase("none", elastic)), ids, 2400.0)
    g = torch.Generator(device="cuda").manual_seed(2)
    eps = 1e-3 * torch.randn((ids.size, 6), generator=g, device="cuda", dtype=torch.float64)
    rate, settings = eps / 1e-4, MaterialUpdateSettings(50, 1.0e-10, 1.0e-12, 1.0e-10)
    needs = MaterialResponseRequirements(tangent=True, free_energy=True, dissipation=True)
    out = model.update(MaterialPointRequest(eps, rate, 1e-4, "three_dimensional", settings), model.initialize_state(ids.size), needs)
    for phase, material in enumerate((j2, elastic)):
        at = torch.as_tensor(np.flatnonzero(ids == phase), device="cuda")
        alone = material.update(MaterialPointRequest(eps[at], rate[at], 1e-4, "three_dimensional", settings),
                                MaterialState(material.initialize_state(at.numel()).variables), needs)  # fmt: skip
        for name in ("stresses", "tangents", "free_energy", "dissipation"):
            assert torch.equal(getattr(out, name)[at], getattr(alone, name)), name
        for name, values in out.diagnostics.items():
            if name in alone.diagnostics:
                assert torch.equal(values[at], alone.diagnostics[name]), name
            elif name not in ("viscoplastic_active", "incremental_work_density", "equivalent_stress_increment"):
                assert bool(torch.isnan(values[at]).all()), name
    outside = torch.as_tensor(np.flatnonzero(ids == 9), device="cuda")
    assert not bool(out.stresses[outside].any()) and not bool(out.tangents[outside].any())
    assert all(bool(torch.isnan(values[outside]).all()) for values in out.diagnostics.values())
