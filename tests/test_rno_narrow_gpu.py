"""GPU tests of the surrogate's narrow window kernels and of the one-launch weight gradients.

The narrow kernels (16 paths per CTA, weights as the MMA's first operand) multiply and add in
the order of the wide ones (128 paths per CTA): a window of few paths must give, bit for bit,
what the same paths give inside a window wide enough for the wide kernels.  The weight
gradients are compared with float64 products of the same bf16 operands: fp32 accumulation of
R <= 1,600 products in at most three K slices is within R eps = 1e-4 of the products'
absolute sum."""

from __future__ import annotations

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

from concrete_impact_b200 import _native  # noqa: E402
from concrete_impact_b200.rno import RNOConfig, RNOSurrogate  # noqa: E402


def _window(rno, paths, steps, data):
    rno.load_window(*(t[:, :paths].contiguous() if t.dim() > 2 or t.shape[0] == steps else t[:paths] for t in data))
    return rno._buffers(steps, paths)


def _data(steps, paths):
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    return r(steps, paths, 6), r(steps, paths, 6), r(steps, paths, 6), 0.05 * torch.rand((steps, paths), generator=g, device="cuda"), r(paths, 6)


@pytest.mark.parametrize("skip", [False, True])
@pytest.mark.parametrize("paths", [1, 8, 15, 16, 17, 130, 2369])
def test_narrow_window_matches_the_wide_one(paths, skip):
    steps = 9
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    wide = 16 * sms * 3 + 16
    data = _data(steps, wide)
    out = []
    for n in (paths, wide):
        rno = RNOSurrogate(RNOConfig(seed=2))
        if skip:
            rno.set_elastic_skip(torch.eye(6).numpy() + 0.1)
        w = _window(rno, n, steps, data)
        c = rno._window_struct(w, True)
        c.loss_scale = 1.0e-3  # the same for both widths
        rno._forward(w, True)
        _native.check(rno.lib.cib_rno_window_backward(ctypes.byref(c), _native.stream_ptr()), "backward")
        assert int(rno.err.item()) == 0
        rows = lambda t: t[:, : n * steps].reshape(t.shape[0], steps, n)[:, :, :paths]  # noqa: E731
        out.append([w["z"][:, :paths], w["gY"][:, :paths], *(z[:, :paths] for z in w["Z"]), rows(w["Xt"]),
                    *(rows(t) for t in w["Ht"]), rows(w["dYt"]), *(rows(t) for t in w["dZt"])])  # fmt: skip
        if n == paths:
            target = w["gY"].double() / (2.0 * 1.0e-3)
            assert float(w["loss_part"].sum()) == pytest.approx(float((target**2).sum()), rel=1e-5)
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("rows,splits", [(64, 1), (512, 1), (1088, 2), (1600, 3)])
def test_weight_gradients_in_one_launch(rows, splits):
    g = torch.Generator(device="cuda").manual_seed(rows)
    shapes = [(128, 32), (128, 128), (128, 128), (16, 128)]
    a = [torch.randn((m, rows), generator=g, device="cuda").to(torch.bfloat16) for m, _ in shapes]
    b = [torch.randn((n, rows), generator=g, device="cuda").to(torch.bfloat16) for _, n in shapes]
    gw = [torch.full(s, 7.0, device="cuda") for s in shapes]
    gb = [torch.full((s[0],), 7.0, device="cuda") for s in shapes]
    partial = torch.empty(splits * sum(m * n for m, n in shapes), device="cuda")
    row_partial = torch.empty(splits * 512, dtype=torch.float64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    c = _native.RNOWgradC()
    c.K, c.ld, c.splits = rows, rows, splits
    for i, (m, n) in enumerate(shapes):
        c.M[i], c.N[i] = m, n
        c.A[i], c.B[i], c.gw[i], c.gb[i] = (t.data_ptr() for t in (a[i], b[i], gw[i], gb[i]))
    c.partial, c.row_partial, c.err = partial.data_ptr(), row_partial.data_ptr(), err.data_ptr()
    lib = _native.load_library()
    _native.check(lib.cib_rno_weight_gradients(ctypes.byref(c), _native.stream_ptr()), "cib_rno_weight_gradients")
    assert int(err.item()) == 0
    for i in range(4):
        exact = a[i].double() @ b[i].double().T
        bound = 1.0e-4 * (a[i].double().abs() @ b[i].double().abs().T)
        assert bool(((gw[i].double() - exact).abs() <= bound).all())
        sums = a[i].double().sum(1)
        assert bool(((gb[i].double() - sums).abs() <= 1.0e-6 * a[i].double().abs().sum(1)).all())
