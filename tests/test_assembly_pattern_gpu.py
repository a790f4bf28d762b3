"""GPU test of the tangents of one assembly cache: each owns its index tensors."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200.assembly import (assemble_hex8_material_response_cached,  # noqa: E402
                                           build_hex8_material_assembly_cache, initialize_hex8_material_state)  # fmt: skip
from concrete_impact_b200.materials import J2ViscoplasticMaterial, MaterialState, MaterialUpdateSettings  # noqa: E402
from concrete_impact_b200.rve import build_structured_hex8_box  # noqa: E402


def test_editing_one_tangents_indices_leaves_the_others() -> None:
    nodes, elements = build_structured_hex8_box((1.0, 1.0, 1.0), (2, 3, 1))
    cache = build_hex8_material_assembly_cache(nodes, elements)
    material = J2ViscoplasticMaterial("mortar", 2200.0, 25.0e9, 0.2, 20.0e6, 2.0e9, 1.0e-3, 20.0e6, 1.0)
    state = initialize_hex8_material_state(material, elements.shape[0])
    state = MaterialState({k: torch.as_tensor(v, device="cuda") for k, v in state.variables.items()})
    u = torch.zeros(3 * nodes.shape[0], dtype=torch.float64, device="cuda")
    settings = MaterialUpdateSettings(50, 1.0e-10, 1.0e-12, 1.0e-10)
    tangents = []
    for _ in range(3):
        k = assemble_hex8_material_response_cached(nodes, elements, material, state, u, u, 1.0e-4, settings, cache).tangent
        np.testing.assert_array_equal(k.crow_indices().cpu().numpy(), cache.csr_indptr)
        np.testing.assert_array_equal(k.col_indices().cpu().numpy(), cache.csr_indices)
        tangents.append(k)
        if len(tangents) == 2:
            k.crow_indices().zero_()
            k.col_indices().zero_()
    np.testing.assert_array_equal(tangents[0].col_indices().cpu().numpy(), cache.csr_indices)
