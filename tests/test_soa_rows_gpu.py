"""GPU tests of the streaming return map on rows at any alignment: the same points in rows that
are 16-byte aligned (padded) and in rows that are not give the same bits, at the edges of a warp's
points and of the rule on points per thread (1,024 per SM)."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import batched  # noqa: E402
from concrete_impact_b200.materials import J2ViscoplasticMaterial, MaterialUpdateSettings  # noqa: E402

MORTAR = J2ViscoplasticMaterial("mortar", 2200.0, 25.0e9, 0.2, 20.0e6, 2.0e9, 1.0e-3, 20.0e6, 1.0)
SETTINGS = MaterialUpdateSettings(50, 1.0e-10, 1.0e-12, 1.0e-10)


def _run(n: int, ld: int, dtype: torch.dtype, rows: int, poison: int | None = None):
    g = torch.Generator(device="cuda").manual_seed(n)
    field = lambda scale: (scale * torch.randn((6, n), generator=g, device="cuda", dtype=torch.float64)).to(dtype)  # noqa: E731
    pad = lambda t: torch.nn.functional.pad(t, (0, ld - n)).contiguous()  # noqa: E731
    de, stress, ep = field(6.0e-4), field(8.0e6), field(1.0e-5)
    eps = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 1e-4
    if poison is not None:
        de[:, poison:] = float("nan")
    old = batched.SoAState(pad(stress), pad(ep), eps)
    new = batched.SoAState(*(torch.full_like(t, 7.0) for t in (old.stress, old.plastic_strain, eps)))
    tangent = torch.full((rows, ld), 7.0, dtype=dtype, device="cuda") if rows else None
    flags = batched._flags(eps.device)
    batched.launch_j2vp_soa(MORTAR, SETTINGS, 1.0e-4, pad(de), old, new, tangent, flags, count=n)
    return new.stress[:, :n], new.plastic_strain[:, :n], new.eqps, tangent[:, :n] if rows else None, int(flags[0])


@pytest.mark.parametrize("rows", [0, 8, 36])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [1, 31, 33, 63, 127, 129, 151_551, 151_553, 300_007])
def test_rows_at_any_alignment(n: int, dtype: torch.dtype, rows: int) -> None:
    odd, even = _run(n, n, dtype, rows), _run(n, (n + 7) // 4 * 4, dtype, rows)
    assert odd[4] == even[4] == -1
    for a, b in zip(odd[:4], even[:4]):
        assert (a is None and b is None) or torch.equal(a, b)


@pytest.mark.parametrize("n, first", [(129, 96), (300_007, 299_999), (300_007, 128)])
def test_the_first_failing_point_is_reported(n: int, first: int) -> None:
    assert _run(n, n, torch.float32, 36, poison=first)[4] == first
