"""GPU test of the layout of a window's loss: row 0 of loss_part holds the sum of squared errors
of each group of 128 paths over the window, the other rows are zero, whichever kernels run."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200.rno import RNOConfig, RNOSurrogate  # noqa: E402


# paths: one tile; a group's last tile and the next group's first; several groups; the narrow
# kernels' most on 148 SMs and the wide ones beyond
@pytest.mark.parametrize("paths, steps", [(5, 8), (128, 8), (129, 9), (700, 50), (300, 7), (7104, 8), (7105, 8)])
def test_row_zero_holds_the_loss_of_every_group(paths: int, steps: int) -> None:
    rno = RNOSurrogate(RNOConfig(seed=2))
    g = torch.Generator(device="cuda").manual_seed(paths)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    rno.load_window(r(steps, paths, 6), r(steps, paths, 6), r(steps, paths, 6),
                    0.05 * torch.rand((steps, paths), generator=g, device="cuda"), r(paths, 6))  # fmt: skip
    w = rno._buffers(steps, paths)
    c = rno._window_struct(w, True)
    c.loss_scale = 0.5  # gS = s - target
    for _ in range(2):
        w["loss_part"].fill_(float("nan"))
        rno._forward(w, True)
        square = (w["gY"].double() ** 2).sum((0, 2))
        groups = torch.stack([part.sum() for part in square.split(128)])
        torch.testing.assert_close(w["loss_part"][0], groups, rtol=1e-12, atol=0.0)  # 128 x 50 x 6 squares in double
        assert not bool(w["loss_part"][1:].any())
    assert int(rno.err.item()) == 0
