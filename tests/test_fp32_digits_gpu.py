"""How far the FP32 kernels are from the FP64 ones on the same inputs: the digits
that FP32 sums and positions have to keep.  Each bound is derived where it
stands."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


def _op(n, na, ns, ds=1.0, start=0.0, **kw):
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    return tc.ParallelProjection2DOp(ns, na, ds, math.pi / na, 0.25, start, n, n, 1.0, 1.0, 0.0, 0.0, **kw)


def _off(f, x):
    """FP32 against FP64 of one call: rel-L2."""
    return rel_l2(host(f(cuda(x))), host(f(cuda(x.astype(np.float64)))))


@pytest.mark.parametrize("n,na,ns", [(64, 90, 95), (130, 100, 190), (300, 64, 500)])
def test_disdriven_grad_noise(n, na, ns):
    """Positions to 2^-24 of a few channels (1.2e-7 rms at most, slopes of 1.4 a
    channel beside terms of 1) and sums of up to 16 views at a time (a few 2^-24):
    3e-7.  Positions to 2^-24 of 60 channels give 5e-7 and more."""
    op = _op(n, na, ns, method="disdriven")
    assert _off(op.adjoint, np.random.default_rng(n).standard_normal((na, ns)).astype(np.float32)) <= 3e-7


@pytest.mark.parametrize("ds", [1.0, 0.3, 0.02, 0.01, 0.0015])
@pytest.mark.parametrize("start", [0.0, 0.4])
def test_disdriven_narrow_channels(ds, start):
    """Footprints down to a thousandth of a pixel, views along the axes (the same
    fraction on every line, so that nothing averages out) and oblique: a line's
    lengths to their own digits, 24 + 4 sums a ray of 96 lines: 4e-7 (2^-24 each,
    all the same way at worst)."""
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    n, na, ns = 96, 16, 120
    op = tc.ParallelProjection2DOp(ns, na, ds, 2 * math.pi / na, 0.25, start, n, n, 1.0, 1.0, 0.3, -0.2, method="disdriven")
    for img in (np.ones((n, n)), np.random.default_rng(2).random((n, n))):
        assert _off(op.forward, img.astype(np.float32)) <= 4e-7


def _ramp(ns, nrow, kind="fan"):
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    return tc.RampFilterOp(ns, nrow, 1.3, 900.0 if kind == "fan" else -1.0, 1 if kind == "fan" else 0)


@pytest.mark.parametrize("ns", [95, 500, 729, 1472, 1537, 2304, 4100])
def test_ramp_phantom(ns):
    """Sinograms of discs: centred sums (the reference input within 8 channels of
    its outputs) of 128 inputs at most, then of these: partial sums about as large
    as the result, sqrt(128 + 16) roundings of 2^-24 = 7e-7 at most.  A reference
    input per 16 outputs gives 9e-7 at 500 channels, sums of 736 inputs 2e-6 at 1472."""
    rng = np.random.default_rng(ns)
    s = np.linspace(-1, 1, ns)[None]
    th = np.linspace(0, math.pi, 48, endpoint=False)[:, None]
    x = 0.01 * rng.standard_normal((48, ns))
    for _ in range(10):
        a, q = rng.uniform(0.05, 0.5), s - rng.uniform(-0.5, 0.5) * np.cos(th + rng.uniform(0, 6))
        x = x + 4 * np.sqrt(np.clip(a * a - q * q, 0, None))
    assert _off(_ramp(ns, 48, "par").forward, x.astype(np.float32)) <= 7e-7


@pytest.mark.parametrize("ns", [5, 96, 185, 729, 1100, 1600, 4096, 4136, 4137, 4700, 5775, 5800])
def test_ramp_same_in_any_batch(ns):
    """A sinogram's result does not depend on those beside it, on either side of
    two CTAs an SM, forward and grad; wide rows against FP64 within 1e-5."""
    import torch
    op = _ramp(ns, 33, "par")
    x = torch.as_tensor(np.random.default_rng(ns).standard_normal((90, 33, ns)).astype(np.float32), device="cuda")
    for f in (op.forward, op.adjoint):
        many = f(x)
        for i in (0, 41, 89):
            assert torch.equal(f(x[i]), many[i])
        if ns > 4000:
            h = np.array([op.taps(x.device).cpu().numpy()]).ravel()
            k = np.arange(ns)
            m = h[ns + k[:, None] - k[None, :]] if f == op.forward else h[ns + k[None, :] - k[:, None]]
            want = 1.3 * (m @ host(x[41]).astype(np.float64).T).T
            assert rel_l2(host(many[41]), want) <= 1e-5


@pytest.mark.parametrize("step", [0.05, 0.125, 0.25, 0.5])
@pytest.mark.parametrize("start", [0.0, 0.013])
def test_ray_casting(step, start):
    """Constant images come out to the last rounding or two (a row's weights add up
    to its samples); discs within the positions' 2^-23 of a pixel at their edges and
    sums of 8 rows, 8 x 2^-25 at worst: 1.5e-7."""
    n = 200
    op = _op(n, 60, 290, start=start, fov=90.0, method="raycasting", step_size=step)
    assert _off(op.forward, np.ones((n, n), np.float32)) <= 1e-7
    y, x = np.mgrid[0:n, 0:n] / n - 0.5
    img = sum(m * ((x - a) ** 2 + (y + a) ** 2 < r) for m, a, r in ((0.02, 0.0, 0.15), (0.013, 0.1, 0.02), (0.03, -0.2, 0.01)))
    assert _off(op.forward, img.astype(np.float32)) <= 1.5e-7


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.3e38])
@pytest.mark.parametrize("method", ["360", "180"])
def test_helical_not_finite(method, value):
    """Infinities and NaN in a scan reach the samples that they reach in FP64, as
    infinities where only measured rows have them (means of rows, 360LI)."""
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    ns, nt, vpr, nz = 130, 16, 300, 24
    cm = nt * 595.0 / 1085.6 / vpr
    op = tc.HelicalInterpolationOp(ns, nt, 4 * vpr, 900.0 / ns, 1.0, 0.375, -0.25, 0.0, 2 * math.pi / vpr, 0.0, cm, vpr, nz,
                                   1.7 * vpr * cm / nz, (vpr + 3.3) * cm, 1.4, 595.0, 1085.6, method)
    rng = np.random.default_rng(5)
    x = rng.random((4 * vpr, nt, ns)).astype(np.float32)
    x[rng.integers(vpr, 3 * vpr, 40), rng.integers(nt, size=40), rng.integers(ns, size=40)] = value
    got, want = host(op.forward(cuda(x))), host(op.forward(cuda(x.astype(np.float64))))
    if value == 3.3e38:
        fine = np.abs(want) < 1e30
        assert rel_l2(got[fine], want[fine]) <= 1e-6
        return
    assert np.array_equal(np.isfinite(got), np.isfinite(want)) and not np.isfinite(want).all()
    fine = np.isfinite(want)
    assert rel_l2(got[fine], want[fine]) <= 1e-6
    if method == "360":
        assert np.array_equal(np.isnan(got), np.isnan(want))
