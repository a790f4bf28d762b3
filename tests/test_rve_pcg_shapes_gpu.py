"""GPU tests of the matrix-free PCG kernel over its shared-memory plans: layer widths from one
element to the widest accepted layer, odd and very flat boxes, every cluster size and block
shape, and tangent arrays that are not aligned for vector loads.

A solve is judged by a strain-displacement operator written with torch in float64, on random
right-hand sides and viscoplastic tangents.  FP64: the solver stops at 1e-11 of the right-hand
side; its recursive residual drifts from the true one by iterations x eps x condition (100 x
1e-16 x 1e3), so 1e-10 is asserted.  FP32: the element products round at 6e-8, which the
condition number of the widest box (about 31^2 x 3) amplifies to 2e-4; 1e-3 is asserted."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200.materials import MaterialUpdateSettings  # noqa: E402
from concrete_impact_b200.rve import LinearSolverOptions, RVEBatch  # noqa: E402
from concrete_impact_b200.rve_builders import build_two_phase_sphere_rve, config0_materials, default_newton  # noqa: E402

SETTINGS = MaterialUpdateSettings(50, 1.0e-10, 1.0e-12, 1.0e-10)
BOXES = [(1, 1, 2), (3, 5, 2), (4, 4, 9), (7, 9, 3), (8, 8, 8), (12, 12, 12), (16, 16, 5), (25, 31, 3), (2, 3, 70)]


def _clusters(divisions, precision):
    """Every accepted cluster size: a z layer per CTA, and a layer within the kernel's range."""
    widest = 711 if precision == 64 else 1066
    return [c for c in (1, 2, 4, 8) if c == 1 or (c <= divisions[2] and divisions[0] * divisions[1] <= widest)]


def _batch(divisions, precision, cluster=1):
    mortar, aggregate = config0_materials()
    model = build_two_phase_sphere_rve(divisions, mortar, aggregate, default_newton(), seed=3)
    batch = RVEBatch([model, model], precision=precision, linear_solver=LinearSolverOptions(cluster=cluster))
    strain = np.random.default_rng(7).standard_normal((2, 6))
    batch.macro.copy_(torch.as_tensor(2.0e-3 * strain))
    batch.dt.fill_(1.0e-5)
    b = batch.batch_struct(SETTINGS)
    batch.residual(b, batch.w, None, None)
    assert int(batch.tflag.sum()) > 0
    rhs = torch.as_tensor(np.random.default_rng(9).standard_normal(3 * batch.nelem), device=batch.device)
    for o in batch.elem_offsets:
        rhs[3 * o : 3 * o + 3] = 0.0
    batch.res.copy_(rhs)
    return batch, b


def _solve(batch, b, rtol):
    batch.pcg(b, batch.res, batch.x, batch.r, batch.p, batch.Ap, batch.nrve, batch.sys_rve, batch.sys_off,
              batch.pcg_status, batch.pcg_iters, batch.pcg_rel, batch.pcg_xnorm, rtol)  # fmt: skip
    assert batch.pcg_status.cpu().tolist() == [0, 0]
    return batch.x.clone()


def _apply(batch, x):
    """K x of both RVEs, from the stored tangent parameters, in float64."""
    model = batch.models[0]
    nx, ny, nz = model.divisions
    h = 1.0 / np.asarray(model.divisions, dtype=float)
    g = 1.0 / np.sqrt(3.0)
    b = np.zeros((8, 6, 24))
    for q in range(8):
        pt = [g if q & bit else -g for bit in (4, 2, 1)]
        for a in range(8):
            s = [1.0 if a & bit else -1.0 for bit in (1, 2, 4)]
            f = [1.0 + s[d] * pt[d] for d in range(3)]
            d = [0.25 * s[0] * f[1] * f[2] / h[0], 0.25 * s[1] * f[0] * f[2] / h[1], 0.25 * s[2] * f[0] * f[1] / h[2]]
            for row, comps in enumerate(((0,), (1,), (2,), (1, 2), (0, 2), (0, 1))):
                if len(comps) == 1:
                    b[q, row, 3 * a + comps[0]] = d[comps[0]]
                else:
                    b[q, row, 3 * a + comps[0]], b[q, row, 3 * a + comps[1]] = d[comps[1]], d[comps[0]]
    bt = torch.as_tensor(b, device=batch.device)
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    nodes = np.stack([((i + (a & 1)) % nx + nx * ((j + (a >> 1 & 1)) % ny + ny * ((k + (a >> 2 & 1)) % nz))).ravel()
                      for a in range(8)], axis=1)  # fmt: skip
    idx = torch.as_tensor(np.concatenate([nodes + o for o in batch.elem_offsets]), device=batch.device)
    dofs = (3 * idx[:, :, None] + torch.arange(3, device=batch.device)).reshape(-1, 24)
    young = torch.tensor([m.young_modulus for _, m in batch.phases], dtype=torch.float64, device=batch.device)
    nu = batch.phases[0][1].poisson_ratio
    e = young[batch.phase.long()][:, None].expand(-1, 8)
    bulk, two_g = e / (3.0 * (1.0 - 2.0 * nu)), e / (1.0 + nu)
    t = batch.tparam.double().T.reshape(-1, 8, 8)
    on = batch.tflag.reshape(-1, 8) > 0
    zero = torch.zeros_like(two_g)
    n = torch.where(on[..., None], t[..., :6], torch.zeros_like(t[..., :6]))
    f, c = torch.where(on, t[..., 6], two_g), torch.where(on, t[..., 7], zero)
    eps = torch.einsum("qij,ej->eqi", bt, x[dofs])
    sig = (0.5 * f)[..., None] * eps + (c * (n * eps).sum(-1))[..., None] * n
    tr = eps[..., :3].sum(-1)
    sig[..., :3] += (0.5 * f)[..., None] * eps[..., :3] + ((bulk - f / 3.0) * tr)[..., None]
    out = torch.zeros_like(x).index_add_(0, dofs.reshape(-1), torch.einsum("qij,eqi->ej", bt, sig).reshape(-1))
    for o in batch.elem_offsets:
        out[3 * o : 3 * o + 3] = 0.0
    return out * float(np.prod(h) / 8.0)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("divisions", BOXES)
def test_solves_the_assembled_system(divisions, precision):
    rtol, bound = (1.0e-11, 1.0e-10) if precision == 64 else (1.0e-6, 1.0e-3)
    for cluster in _clusters(divisions, precision):
        batch, b = _batch(divisions, precision, cluster)
        for shape in (0, 1, 2, 3):
            batch.pcg_shape = shape
            left = float((_apply(batch, _solve(batch, b, rtol)) - batch.res).norm() / batch.res.norm())
            assert left <= bound, (cluster, shape, left)


@pytest.mark.parametrize("divisions", [(3, 5, 2), (8, 8, 8), (12, 12, 12), (25, 31, 3), (2, 3, 70)])
def test_fp64_solution_does_not_depend_on_the_launch(divisions):
    """The same bits for every cluster size and block shape."""
    reference = None
    for cluster in _clusters(divisions, 64):
        batch, b = _batch(divisions, 64, cluster)
        for shape in (0, 1, 2, 3):
            batch.pcg_shape = shape
            x = _solve(batch, b, 1.0e-11)
            reference = x if reference is None else reference
            assert torch.equal(x, reference), (cluster, shape)


@pytest.mark.parametrize("precision", [64, 32])
def test_unaligned_tangent_parameters(precision):
    batch, b = _batch((5, 4, 4), precision, 2)
    rtol = 1.0e-11 if precision == 64 else 1.0e-6
    aligned = _solve(batch, b, rtol)
    shifted = torch.empty(batch.tparam.numel() + 1, dtype=batch.tparam.dtype, device=batch.device)[1:]
    shifted.copy_(batch.tparam.reshape(-1))
    assert shifted.data_ptr() % 16 != 0
    b.tparam = shifted.data_ptr()
    assert torch.equal(_solve(batch, b, rtol), aligned)
