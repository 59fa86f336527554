"""Helical rebinning in FP32 by groups of channels, views and slices, against the
oracle port: channels, views and slices around the groups' sizes, slabs from less
than a row to many rows, pitches with one and two samples on the detector.

Tolerance: 2e-6 of the output's peak (a wrong row or view would move a value by
O(0.1))."""
import numpy as np
import pytest

from gpu_helpers import cuda, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["360", "180"])
@pytest.mark.parametrize("ns,nt,vpr,nz,pitch,thickness", [
    (31, 8, 37, 3, 1.0, 0.3), (32, 16, 64, 8, 1.0, 1.0), (33, 16, 66, 9, 0.6, 2.0), (127, 32, 131, 17, 0.9, 6.0),
    (129, 12, 200, 5, 1.0, 0.0), (200, 64, 97, 20, 0.45, 1.25),
    (290, 16, 330, 20, 1.0, 1.0), (321, 20, 257, 23, 0.8, 2.5), (257, 16, 300, 24, 0.9, 0.0)])
def test_helical_groups(port, method, ns, nt, vpr, nz, pitch, thickness):
    _check(port, method, ns, nt, vpr, nz, pitch, thickness, 1.0)


@pytest.mark.parametrize("method", ["360", "180"])
@pytest.mark.parametrize("ns,nt,vpr,nz,pitch,thickness", [
    (290, 16, 330, 20, 1.0, 1.0), (321, 20, 257, 23, 0.8, 2.5), (257, 16, 300, 24, 0.9, 0.0), (300, 24, 400, 24, 0.5, 1.4)])
def test_helical_couch_backwards(port, method, ns, nt, vpr, nz, pitch, thickness):
    """The slab's rows move the other way from view to view."""
    _check(port, method, ns, nt, vpr, nz, pitch, thickness, -1.0)


def _check(port, method, ns, nt, vpr, nz, pitch, thickness, sign):
    from oracle import Heli
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    dso, dsd = 595.0, 1085.6
    cm = sign * pitch * nt * dso / dsd / vpr
    na = 4 * vpr
    h = Heli.make(ns=ns, nt=nt, na=na, ds=900.0 / ns, dt=1.0, view_per_rot=vpr, couch_mov=cm, nz=nz,
                  dz=1.7 * vpr * cm / nz, z0=(vpr + 3.3) * cm, thickness=thickness, dso=dso, dsd=dsd, offset_s=0.375,
                  offset_t=-0.25)
    op = tc.HelicalInterpolationOp(h.ns, h.nt, h.na, h.ds, h.dt, h.offset_s, h.offset_t, h.orbit_start, h.orbit,
                                   h.couch_begin, h.couch_mov, h.view_per_rot, h.nz, h.dz, h.z0, h.thickness, h.dso,
                                   h.dsd, method)
    x = np.random.default_rng(ns + nz).random((2, na, nt, ns)).astype(np.float32)
    got = host(op.forward(cuda(x)))
    for b in range(2):
        want, outside = port.helical(x[b], h, method)
        assert not outside
        assert np.abs(got[b] - want).max() <= 2e-6 * np.abs(want).max()
        assert np.array_equal(got[b], host(op.forward(cuda(x[b]))))
