"""GPU tests of the persistent CSR PCG (one launch per solve, one or six right-hand sides) at the
edges of its partition of rows over CTAs and of the rules that leave a system to the launch per
phase, against float64 residuals and a sparse direct solve."""

from __future__ import annotations

import numpy as np
import pytest
import torch
from scipy.sparse import csr_matrix, diags, random as sparse_random
from scipy.sparse.linalg import spsolve

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import _native  # noqa: E402
from concrete_impact_b200.rve_general import _ReducedSystem  # noqa: E402

RTOL = 1.0e-11


def _matrix(n: int, kind: str) -> csr_matrix:
    """Symmetric, diagonally dominant by 5 %; rows of 1 to 5 entries (band), up to 81 in a row of
    neighbours (wide) or anywhere (scattered: many columns per CTA)."""
    rng = np.random.default_rng(n)
    if kind == "band":
        a = diags([rng.uniform(-1, 1, n - k) * (rng.random(n - k) < 0.8) for k in (1, 7)], [1, 7], (n, n), format="csr")
    elif kind == "wide":
        a = diags([rng.uniform(-1, 1, n - k) for k in range(1, 41)], range(1, 41), (n, n), format="csr")
    else:
        a = sparse_random(n, n, 40.0 / n, "csr", random_state=n, data_rvs=lambda k: rng.uniform(-1, 1, k))
    a = (a + a.T).tocsr()
    a.setdiag(0.0)
    a.eliminate_zeros()
    a = (a + diags(1.05 * np.asarray(abs(a).sum(1)).ravel() + rng.uniform(0.5, 2.0, n))).tocsr()
    a.sort_indices()
    return a


def _system(a: csr_matrix, maxit: int = 2000) -> _ReducedSystem:
    dev = _native.require_cuda()
    system = _ReducedSystem(a.indptr, a.indices, a.shape[0], dev, RTOL, maxit)
    system.prepare(_native.load_library(), torch.as_tensor(a.data, device=dev))
    return system


# Rows: below the smallest system taken, that one, ragged last CTAs around 18 rows each on 148
# SMs, the largest system taken and one more; and one whose CTAs touch too many columns to fit.
@pytest.mark.parametrize("n, kind", [(63, "band"), (64, "band"), (65, "wide"), (145, "wide"), (2664, "wide"), (2665, "band"),
                                     (5000, "scattered"), (28416, "band"), (28417, "band"), (20000, "scattered")])  # fmt: skip
def test_solves_meet_their_residual_and_repeat(n: int, kind: str) -> None:
    a, lib = _matrix(n, kind), _native.load_library()
    system = _system(a)
    b = np.random.default_rng(1).standard_normal((6, n)) * np.array([1.0, 1e-6, 1e8, 1.0, 1.0, 1.0])[:, None]
    b[3] = 0.0
    b[4, n // 2 :] = 0.0
    rhs = torch.as_tensor(b, device="cuda")
    six, status = system.solve_six(lib, rhs)
    assert status == [0] * 6 and torch.equal(six, system.solve_six(lib, rhs)[0])
    assert not bool(six[3].any())
    # ||b - A x|| beside the recurrence's residual: a rounding per entry of a row and iteration,
    # |A| |x| <= 3 ||b|| for this dominance, at most 500 iterations
    tol = RTOL + 3.0 * (81 + 500) * 2.0**-53 * 2.0
    for j in (0, 1, 2, 4, 5):
        x, one, iterations, rel = system.solve(lib, rhs[j])
        assert one == 0 and 0 < iterations <= 500 and rel <= RTOL
        for got in (x, six[j]):
            assert np.linalg.norm(b[j] - a @ got.cpu().numpy()) <= tol * np.linalg.norm(b[j]), j
    if n < 3000:
        exact = spsolve(a.tocsc(), b[0])
        assert np.linalg.norm(six[0].cpu().numpy() - exact) <= 50 * tol * np.linalg.norm(exact)  # cond <= 42


def test_iteration_limit_and_breakdown() -> None:
    a, lib = _matrix(500, "wide"), _native.load_library()
    rhs = torch.ones((6, 500), dtype=torch.float64, device="cuda")
    rhs[1] = 0.0
    system = _system(a, maxit=2)
    before = system.iterations
    _, status = system.solve_six(lib, rhs)
    assert status == [1, 0, 1, 1, 1, 1] and system.iterations - before == 10
    _, status, iterations, rel = system.solve(lib, rhs[0])
    assert status == 1 and iterations == 2 and rel > RTOL
    system = _system(a, maxit=0)
    assert system.solve(lib, rhs[0])[1:3] == (1, 0)
    system = _system((a - 2.0 * diags(a.diagonal())).tocsr())  # negative diagonal: p.Ap < 0
    assert system.solve(lib, rhs[0])[1] == 2
    rhs[0, 7] = float("nan")
    _, status = _system(a).solve_six(lib, rhs)
    assert status == [2, 0, 0, 0, 0, 0]
