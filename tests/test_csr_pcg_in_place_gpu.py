"""GPU tests of cib_csr_pcg and cib_csr_pcg_block with the right-hand side in the array of the
solution or of a scratch vector, for systems that the persistent solve takes, refuses by size and
gives back because some CTAs' rows do not fit."""

from __future__ import annotations

import ctypes
import functools

import numpy as np
import pytest
import torch
from scipy.sparse import block_diag, csr_matrix, diags

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import _native  # noqa: E402
from test_csr_pcg_grid_gpu import _matrix, _system  # noqa: E402

RTOL = 1.0e-11


@functools.cache
def _half_scattered(n: int) -> csr_matrix:
    """Rows of a few neighbours in the first half; some 120 columns anywhere to a row in the
    second, whose CTAs give the solve back (190 rows of 28,000 at 10 bytes an entry)."""
    m = n // 2
    rng = np.random.default_rng(n)
    a = csr_matrix((rng.uniform(-1, 1, 60 * m), (np.repeat(np.arange(m), 60), rng.integers(0, m, 60 * m))), (m, m))
    a = (a + a.T).tocsr()
    a.setdiag(0.0)
    a = a + diags(1.05 * np.asarray(abs(a).sum(1)).ravel() + rng.uniform(0.5, 2.0, m))
    a = block_diag([_matrix(m, "band"), a], "csr")
    a.sort_indices()
    return a


CASES = [(63, "band"), (500, "wide"), (28000, "half"), (28417, "band")]


def _setup(n: int, kind: str):
    a = _half_scattered(n) if kind == "half" else _matrix(n, kind)
    return a, _system(a)


@pytest.mark.parametrize("where", ["x", "r", "z", "p", "q"])
@pytest.mark.parametrize("n, kind", CASES)
def test_right_hand_side_in_another_array_of_the_call(n: int, kind: str, where: str) -> None:
    a, s = _setup(n, kind)
    b = np.random.default_rng(1).standard_normal(n)
    v = {name: torch.empty(n, dtype=torch.float64, device="cuda") for name in "xrzpq"}
    v[where].copy_(torch.as_tensor(b))
    status, iterations, rel = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_double()
    _native.check(_native.load_library().cib_csr_pcg(
        n, s.indptr.data_ptr(), s.indices.data_ptr(), s.values.data_ptr(), s.free.data_ptr(), s.dinv.data_ptr(),
        v[where].data_ptr(), *(v[k].data_ptr() for k in "xrzpq"), s.work.data_ptr(), RTOL, 2000, 16,
        ctypes.byref(status), ctypes.byref(iterations), ctypes.byref(rel), _native.stream_ptr()), "cib_csr_pcg")  # fmt: skip
    assert status.value == 0 and iterations.value > 0
    # as in test_csr_pcg_grid_gpu, with rows of at most 200 entries
    tol = RTOL + 3.0 * (200 + 500) * 2.0**-53 * 2.0
    assert np.linalg.norm(b - a @ v["x"].cpu().numpy()) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("n, kind", CASES)
def test_six_right_hand_sides_in_the_array_of_the_solutions(n: int, kind: str) -> None:
    a, s = _setup(n, kind)
    b = np.random.default_rng(1).standard_normal((6, n))
    b[3] = 0.0
    x = torch.as_tensor(b, device="cuda").clone()
    work = torch.empty(12 * n + 24576, dtype=torch.float64, device="cuda")
    status, iterations, rel = (ctypes.c_int32 * 6)(), (ctypes.c_int32 * 6)(), (ctypes.c_double * 6)()
    _native.check(_native.load_library().cib_csr_pcg_block(
        n, s.indptr.data_ptr(), s.indices.data_ptr(), s.values.data_ptr(), s.free.data_ptr(), s.dinv.data_ptr(),
        x.data_ptr(), x.data_ptr(), work.data_ptr(), RTOL, 2000, 16, status, iterations, rel, _native.stream_ptr()),
        "cib_csr_pcg_block")  # fmt: skip
    assert list(status) == [0] * 6 and not bool(x[3].any())
    tol = RTOL + 3.0 * (200 + 500) * 2.0**-53 * 2.0
    for j in (0, 1, 2, 4, 5):
        assert np.linalg.norm(b[j] - a @ x[j].cpu().numpy()) <= tol * np.linalg.norm(b[j]), j
