"""GPU tests of the choice of the RVE PCG's launch: one CTA per system is the same solve whatever
the shape bits."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from test_rve_pcg_shapes_gpu import _batch, _solve  # noqa: E402


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("divisions", [(8, 8, 8), (12, 12, 12), (25, 31, 3)])
def test_shape_bits_do_not_change_a_solve_on_one_cta(divisions, precision) -> None:
    batch, b = _batch(divisions, precision)
    solutions = []
    for shape in (0, 1, 2, 3):
        batch.pcg_shape = shape
        solutions.append((_solve(batch, b, 1.0e-6), batch.pcg_iters.cpu().tolist()))
    for x, iterations in solutions[1:]:
        assert torch.equal(x, solutions[0][0]) and iterations == solutions[0][1]
