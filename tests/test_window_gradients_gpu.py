"""GPU tests of split-K products whose columns do not fill every slice: the partial tiles that
cib_mlp_gemm hands to cib_splitk_reduce."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import mlp  # noqa: E402


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
