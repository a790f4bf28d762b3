"""GPU tests of the choice of the RVE PCG's launch: one CTA per system is the same solve whatever
the shape bits, the number of systems, which decides over the CTAs of each, changes none, and a
stored choice counts for the kernels that it was measured on."""

from __future__ import annotations

import json

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import rve as R  # noqa: E402
from concrete_impact_b200.rve import LinearSolverOptions, RVEBatch  # noqa: E402
from concrete_impact_b200.rve_builders import build_two_phase_sphere_rve, config0_materials, default_newton  # noqa: E402
from test_rve_pcg_shapes_gpu import SETTINGS, _batch, _solve  # noqa: E402


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


# systems: on 148 SMs the last numbers with 8, 4 and 2 CTAs each and one beyond, in one turn of
# clusters and in whole SMs.  FP32 takes the CTAs that it is asked for, and other shared-memory
# plans from 149 CTAs on.
@pytest.mark.parametrize("systems", [15, 16, 18, 19, 33, 34, 37, 38, 74, 75, 149])
@pytest.mark.parametrize("precision, cluster", [(64, 1), (64, 2), (32, 1), (32, 4)])
def test_solve_does_not_depend_on_the_systems_beside_it(systems: int, precision: int, cluster: int) -> None:
    mortar, aggregate = config0_materials()
    model = build_two_phase_sphere_rve((4, 3, 5), mortar, aggregate, default_newton(), seed=3)
    strain = torch.as_tensor(2.0e-3 * np.random.default_rng(7).standard_normal((systems, 6)))

    def solve(which: list[int], ctas: int) -> torch.Tensor:
        batch = RVEBatch([model] * len(which), precision=precision, linear_solver=LinearSolverOptions(cluster=ctas))
        batch.macro.copy_(strain[which])
        batch.dt.fill_(1.0e-5)
        b = batch.batch_struct(SETTINGS)
        batch.residual(b, batch.w, None, None)
        batch.pcg(b, batch.res, batch.x, batch.r, batch.p, batch.Ap, batch.nrve, batch.sys_rve, batch.sys_off,
                  batch.pcg_status, batch.pcg_iters, batch.pcg_rel, batch.pcg_xnorm, 1.0e-11 if precision == 64 else 1.0e-6)  # fmt: skip
        assert batch.pcg_status.cpu().tolist() == [0] * len(which)
        return batch.x.reshape(len(which), -1).clone()

    together = solve(list(range(systems)), cluster)
    for i in (0, systems // 2, systems - 1):
        assert torch.equal(solve([i], cluster if precision == 32 else 1)[0], together[i]), i


@pytest.mark.parametrize("precision", [64, 32])
def test_stored_choice_of_other_kernels_is_measured_again(tmp_path, monkeypatch, precision) -> None:
    path = tmp_path / "tuning.json"
    monkeypatch.setenv("CIB_TUNING_CACHE", str(path))
    batch, _ = _batch((5, 4, 4), precision, 2)
    # the key without a version, as it was stored for kernels whose shapes meant other launches
    old = f"f{precision}|{torch.cuda.get_device_name(batch.device)}|5x4x4:2"
    path.write_text(json.dumps({old: {"cluster": 4, "shape": 3, "ms": {}}}))
    first = R.tune_pcg_cluster(batch, SETTINGS)
    assert not first["cached"] and first["key"] != old
    assert set(first["ms"]) == {"1/0"} | {f"{c}/{s}" for c in (2, 4) for s in range(4)}
    assert old in json.loads(path.read_text())  # other entries stay
    again = R.tune_pcg_cluster(batch, SETTINGS)
    assert again["cached"] and (again["cluster"], again["shape"]) == (first["cluster"], first["shape"])
