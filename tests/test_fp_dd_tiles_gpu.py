"""The FP32 distance-driven projector and its grad against the oracle: image
sides around the grad's 32 x 64 tiles and the projector's groups of lines,
detectors shorter than the image (footprints cut at the first channel, and past
the last one), footprints of one to many pixels, pixels of one to many channels,
anisotropic pixels, all directions, infinities.

Tolerance: the FP32 parity bound of the projectors (rel-L2 1e-5)."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


def _case(n, ns, na, ds, dx=1.0, dy=1.0, start=0.05):
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    g = dict(ns=ns, na=na, ds=ds, orbit=2 * math.pi / na, offset_s=0.3, orbit_start=start, nx=n, ny=n, dx=dx, dy=dy,
             offset_x=0.25, offset_y=-0.6, fov=-1.0)
    return Geom.make(**g), tc.ParallelProjection2DOp(*g.values(), method="disdriven")


@pytest.mark.parametrize("n,ns,na,ds,dx,dy", [
    (2, 5, 7, 1.0, 1.0, 1.0), (31, 50, 15, 1.0, 1.0, 1.0), (32, 30, 16, 1.0, 1.0, 1.0), (33, 64, 17, 1.3, 1.0, 0.8),
    (64, 65, 33, 0.7, 1.0, 1.0), (65, 40, 40, 1.0, 0.9, 1.1), (97, 200, 50, 0.5, 1.0, 1.0), (70, 20, 20, 3.1, 1.0, 1.0),
    (40, 300, 12, 0.2, 1.0, 1.0), (130, 190, 300, 1.0, 1.0, 1.0)])
def test_disdriven(port, n, ns, na, ds, dx, dy):
    g, op = _case(n, ns, na, ds, dx, dy)
    rng = np.random.default_rng(n + ns)
    img = rng.random((2, n, n)).astype(np.float32)
    proj = rng.standard_normal((2, na, ns)).astype(np.float32)
    fwd, grad = host(op.forward(cuda(img))), host(op.adjoint(cuda(proj)))
    for b in range(2):
        assert rel_l2(fwd[b], port.fp_par_2d_dd(img[b], g)) <= 1e-5
        assert rel_l2(grad[b], port.fp_par_2d_dd_grad(proj[b], g)) <= 1e-5
        assert np.array_equal(fwd[b], host(op.forward(cuda(img[b]))))
        assert np.array_equal(grad[b], host(op.adjoint(cuda(proj[b]))))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3e38])
def test_disdriven_not_finite(port, value):
    """One such pixel or channel reaches the same results as in the oracle."""
    g, op = _case(48, 75, 24, 1.0)
    rng = np.random.default_rng(3)
    img = rng.random((48, 48)).astype(np.float32)
    proj = rng.random((24, 75)).astype(np.float32)
    img[20, 31] = value
    proj[5, 40] = value
    for got, want in ((host(op.forward(cuda(img))), port.fp_par_2d_dd(img, g)),
                      (host(op.adjoint(cuda(proj))), port.fp_par_2d_dd_grad(proj, g))):
        fine = np.isfinite(want) & (np.abs(want) < 1e30)
        assert np.array_equal(fine, np.isfinite(got) & (np.abs(got) < 1e30))
        assert rel_l2(got[fine], want[fine]) <= 1e-5


@pytest.mark.parametrize("n,ns,na,ds,orbit,start", [
    (300, 301, 33, 0.7, 1.0, math.pi / 2), (64, 301, 8, 1.0, -math.pi / 8, 0.0), (300, 33, 91, 0.7, 1.0, math.pi / 2),
    (130, 64, 120, 0.7, -0.02, 0.1)])
def test_disdriven_grad_unfolded_angles(port, n, ns, na, ds, orbit, start):
    """Views below 0 and beyond 2 pi, whose lines may run across the channels:
    footprints far narrower than a channel with weights to match.  Every pixel
    within 1e-5 of the peak (fixed point to 2^-24 of a channel, a few dozen times
    the usual weight)."""
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    g = dict(ns=ns, na=na, ds=ds, orbit=orbit, offset_s=0.25, orbit_start=start, nx=n, ny=n, dx=0.9, dy=0.9,
             offset_x=-4.25, offset_y=1.1, fov=-1.0)
    proj = np.random.default_rng(n + ns).standard_normal((na, ns)).astype(np.float32)
    got = host(tc.ParallelProjection2DOp(*g.values(), method="disdriven").adjoint(cuda(proj)))
    want = port.fp_par_2d_dd_grad(proj, Geom.make(**g))
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
