"""Single-view backprojection (FP32) where rows leave the detector: images wider
than it, views along the axes whose pixels lie exactly on a detector's end, wide
launches with shared sectors.  The pixels outside are exactly the oracle's, the
others within the parity bound (rel-L2 1e-5), those in the end channels to the
digits of two floats (2e-7 of the largest)."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


def _case(n, na, ns, ds, offset, start, orbit, seed=0):
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    g = dict(ns=ns, na=na, ds=ds, orbit=orbit, offset_s=offset, orbit_start=start, nx=n, ny=n, dx=1.0, dy=1.0,
             offset_x=0.0, offset_y=0.0, fov=-1.0)
    x = np.random.default_rng(n + ns + seed).random((na, ns)).astype(np.float32) + 0.5
    return tc.ParallelBackprojection2DOp(*g.values()), Geom.make(**g), x


@pytest.mark.parametrize("n,na,ns,ds,offset,start,orbit", [
    (64, 33, 40, 1.0, 0.0, 0.013, 0.1), (65, 40, 41, 1.0, 0.0, 0.0, math.pi / 2), (96, 8, 63, 1.0, 0.5, 0.0, math.pi / 2),
    (130, 31, 3, 0.7, 0.0, 0.2, 0.1), (200, 45, 150, 0.37, 20.0, 0.0, 0.15), (260, 41, 200, 1.3, -3.0, 0.0, -0.07)])
def test_rows_past_the_detector(port, n, na, ns, ds, offset, start, orbit):
    op, g, x = _case(n, na, ns, ds, offset, start, orbit)
    want = port.bp_par_2d_sv(x, g)
    got = host(op.single_view(cuda(x))).reshape(want.shape)
    assert np.array_equal(got == 0, want == 0)  # x > 0: what is outside
    assert rel_l2(got, want) <= 1e-5
    # pixels between the first or last two channels
    s = host(op.single_view(cuda(np.broadcast_to(np.arange(ns, dtype=np.float64), (na, ns)).copy()))).reshape(want.shape)
    ends = (want != 0) & ((s < 1) | (s > ns - 2))
    assert np.abs(got - want)[ends].max() <= 2e-7 * 1.5 + 1e-7


@pytest.mark.parametrize("na", [704, 705, 708, 713])
def test_bands(port, na):
    """Outputs beyond L2 and within it, whole and shared sectors: an image is the
    same by itself and in a batch (other bands of rows)."""
    import torch
    op, g, x = _case(160, na, 220, 1.0, 0.0, 0.0, math.pi / na)
    xs = torch.stack([cuda(x), 2 * cuda(x), cuda(x)])
    got = op.single_view(xs)
    assert torch.equal(got[0], op.single_view(cuda(x)).reshape(got[0].shape)) and torch.equal(got[2], got[0]) and torch.equal(got[1], 2 * got[0])
    assert rel_l2(host(got[0]), port.bp_par_2d_sv(x, g)) <= 1e-5
