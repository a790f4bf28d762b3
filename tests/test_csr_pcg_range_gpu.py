"""GPU test of cib_csr_pcg on right-hand sides near the ends of the number range, whose dot products
underflow or come near it: the solution scales with the right-hand side."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import _native  # noqa: E402
from test_csr_pcg_grid_gpu import _matrix, _system  # noqa: E402


# 2^-498 (1e-150): r.r ends at 1e-322, where a number has one or two digits; 2^-440 (3.5e-133) and
# 2^500: far enough from the ends that every rounding is that of the unscaled solve
@pytest.mark.parametrize("n", [64, 500, 5000])
@pytest.mark.parametrize("power, rtol, bound", [(-498, 1.0e-10, 1.0e-6), (-440, 1.0e-11, 0.0), (500, 1.0e-11, 0.0)])
def test_solution_scales_with_the_right_hand_side(n: int, power: int, rtol: float, bound: float) -> None:
    system, lib = _system(_matrix(n, "wide" if n > 80 else "band")), _native.load_library()
    system.rtol = rtol
    b = torch.randn(n, dtype=torch.float64, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    want, status, iterations, _ = system.solve(lib, b)
    assert status == 0
    scale = 2.0**power
    x, status, count, rel = system.solve(lib, b * scale)
    assert status == 0 and rel <= rtol
    assert float((x / scale - want).norm() / want.norm()) <= bound
    if bound == 0.0:
        assert count == iterations
    six, codes = system.solve_six(lib, torch.stack([b * scale] * 6))
    assert codes == [0] * 6 and float((six / scale - want).norm() / want.norm()) <= (bound or 1.0e-9)
