"""GPU tests of split-K products whose columns do not fill every slice: the partial tiles that
cib_mlp_gemm hands to cib_splitk_reduce, and the weight gradients of surrogate windows."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import mlp  # noqa: E402
from concrete_impact_b200.rno import RNOConfig, RNOSurrogate  # noqa: E402


@pytest.mark.parametrize("m, k, splits", [(16, 832, 12), (128, 64, 5), (300, 15040, 29)])
def test_every_slice_of_a_split_product_is_written(m: int, k: int, splits: int) -> None:
    """Slices are cut at multiples of 64 columns, so fewer than ``splits`` can hold any: the
    others are zero.  fp32 sums of k products: within k 2^-23 of the products' absolute sum."""
    g = torch.Generator(device="cuda").manual_seed(k)
    a, b = (torch.randn((r, k), generator=g, device="cuda").to(torch.bfloat16) for r in (m, 48))
    partial = torch.full((splits, m, 48), float("nan"), device="cuda")
    out, err = torch.empty((m, 48), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    mlp.gemm(mlp.EPI_PARTIAL, a, b, c=partial.view(splits * m, 48), splits=splits, err=err)
    mlp.splitk_reduce(partial, splits, m, 48, out)
    assert int(err.item()) == 0
    exact, size = a.double() @ b.double().T, a.double().abs() @ b.double().abs().T
    assert bool(((out.double() - exact).abs() <= k * 2.0**-23 * size).all())


@pytest.mark.parametrize("paths, steps, hidden", [(300, 50, 128), (464, 50, 128), (768, 25, 128), (1000, 25, 128),
                                                  (1024, 50, 128), (512, 50, 128), (300, 50, 64), (50, 6, 16), (7, 1, 128)])  # fmt: skip
def test_window_gradients_are_the_products_of_their_operands(paths: int, steps: int, hidden: int) -> None:
    """All four layers against float64 products of the window's own bf16 operands, twice in a row
    (the second time over what the first left in the work buffers).  A slice of at most 1,024
    columns is 64 steps of the tensor core, each rounding its sum at 2^-22; up to 64 slices, whose
    sum may be an eighth of their sizes', are added with 2^-24 each: 64 2^-22 8 + 64 2^-24 8 =
    1.6e-4 of the gradient's norm.  (Slices that were never written put the last layer off by
    2e-3 to 5e-3.)  Bias gradients are sums in double: 2^-23."""
    rno = RNOSurrogate(RNOConfig(seed=2, hidden=hidden))
    g = torch.Generator(device="cuda").manual_seed(paths)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    for _ in range(2):
        rno.load_window(r(steps, paths, 6), r(steps, paths, 6), r(steps, paths, 6),
                        0.05 * torch.rand((steps, paths), generator=g, device="cuda"), r(paths, 6))  # fmt: skip
        rno.window_gradients(steps, paths)
        w = rno._window
        assert int(rno.err.item()) == 0
        pairs = zip([*w["dZt"], w["dYt"]], [w["Xt"], *w["Ht"]], rno.layers)
        for i, (a, b, layer) in enumerate(pairs):
            exact = a.double() @ b.double().T
            assert float((layer.gw.double() - exact).norm() / exact.norm()) <= 1.6e-4, i
            bound = 2.0**-23 * a.double().abs().sum(1)
            assert bool(((layer.gb.double() - a.double().sum(1)).abs() <= bound).all()), i
