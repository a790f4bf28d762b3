"""GPU tests of periodic boxes of a single z layer, whose linear solve has one owner whatever
number of CTAs the launch gives a system: alone, beside thicker boxes in one batch, and through
the whole equilibrium solve.  Tolerances of the linear solves as in test_rve_pcg_shapes_gpu; the
equilibrium solve against the oracle's direct-solve Newton as in test_rve_gpu (1e-6)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import rve as R  # noqa: E402
from concrete_impact_b200.rve_builders import build_two_phase_sphere_rve, config0_materials, default_newton  # noqa: E402
from oracle import j2vp as oj  # noqa: E402
from oracle.rve import OraclePhase, OracleRVE, RVEOracle  # noqa: E402
from test_rve_pcg_shapes_gpu import SETTINGS, _apply, _batch, _solve  # noqa: E402


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("divisions", [(8, 8, 1), (3, 5, 1), (1, 2, 1), (25, 31, 1)])
def test_one_layer_solves_the_assembled_system(divisions, precision):
    rtol, bound = (1.0e-11, 1.0e-10) if precision == 64 else (1.0e-6, 1.0e-3)
    batch, b = _batch(divisions, precision)
    reference = None
    for shape in (0, 1, 2, 3):
        batch.pcg_shape = shape
        x = _solve(batch, b, rtol)
        left = float((_apply(batch, x) - batch.res).norm() / batch.res.norm())
        assert left <= bound, (shape, left)
        if precision == 64:
            reference = x if reference is None else reference
            assert torch.equal(x, reference), shape


@pytest.mark.parametrize("precision", [64, 32])
def test_one_layer_beside_thicker_boxes(precision):
    """The bits of every RVE's solve are those of a batch of this RVE alone.  (1, 1, 1) has one
    node, which is the fixed one: a zero right-hand side."""
    mortar, aggregate = config0_materials()
    models = [build_two_phase_sphere_rve(d, mortar, aggregate, default_newton(), seed=3)
              for d in ((8, 8, 1), (4, 4, 5), (1, 1, 1), (8, 8, 8), (3, 5, 1))]  # fmt: skip
    strain = torch.as_tensor(2.0e-3 * np.random.default_rng(7).standard_normal((len(models), 6)))
    rtol = 1.0e-11 if precision == 64 else 1.0e-6

    def solve(which):
        batch = R.RVEBatch([models[i] for i in which], precision=precision)
        batch.macro.copy_(strain[which])
        batch.dt.fill_(1.0e-5)
        b = batch.batch_struct(SETTINGS)
        batch.residual(b, batch.w, None, None)
        batch.pcg(b, batch.res, batch.x, batch.r, batch.p, batch.Ap, batch.nrve, batch.sys_rve, batch.sys_off,
                  batch.pcg_status, batch.pcg_iters, batch.pcg_rel, batch.pcg_xnorm, rtol)  # fmt: skip
        assert batch.pcg_status.cpu().tolist() == [0] * len(which)
        at = np.concatenate([[0], np.cumsum(3 * batch.elem_counts)])
        return [batch.x[at[k] : at[k + 1]].clone() for k in range(len(which))], batch.pcg_iters.cpu().tolist()

    together, iterations = solve(list(range(len(models))))
    for i, x in enumerate(together):
        alone, one = solve([i])
        assert torch.equal(x, alone[0]) and iterations[i] == one[0], models[i].divisions
    assert not bool(together[2].any()) and min(iterations[:2] + iterations[3:]) > 0


def test_one_layer_equilibrium_matches_the_oracle():
    divisions = (6, 5, 1)
    mortar, aggregate = config0_materials()
    model = build_two_phase_sphere_rve(divisions, mortar, aggregate, default_newton(), seed=3)
    assert set(np.unique(model.element_phase_ids)) == {0, 1}
    macro = np.array([-2.0e-3, 5.0e-4, 5.0e-4, 2.0e-4, 1.0e-4, -3.0e-4])
    got = R.solve_rve_microequilibrium(model, R.RVERequest(macro, 1.0e-4, SETTINGS), R.initialize_rve_state(model))
    ns = model.newton_settings
    names = ("max_iterations", "residual_absolute_tolerance", "residual_relative_tolerance",
             "increment_absolute_tolerance", "increment_relative_tolerance")  # fmt: skip
    oracle = RVEOracle(OracleRVE(divisions, (1.0, 1.0, 1.0),
                                 [OraclePhase("j2", oj.mortar_params()), OraclePhase("elastic", None, 50.0e9, 0.2)],
                                 model.element_phase_ids.astype(np.int64),
                                 {**{name: getattr(ns, name) for name in names}, "armijo": None}))  # fmt: skip
    want = oracle.solve(macro, 1.0e-4, oracle.initial_state(), True)
    for name in ("macro_stress", "effective_tangent"):
        a, b = np.asarray(getattr(got, name)), np.asarray(want[name])
        assert np.abs(a - b).max() <= 1.0e-6 * np.abs(b).max(), name
