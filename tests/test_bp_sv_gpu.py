"""Single-view backprojection (FP32) against the oracle: view counts around the
groups of 32, image rows around the bands, odd widths and segments, pixels of a
fraction of a channel to several channels, all directions.

Tolerance: the FP32 parity bound (rel-L2 1e-5)."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,na,ns,ds", [
    (1, 1, 1, 3, 1.0), (63, 5, 31, 120, 1.0), (64, 33, 32, 99, 1.0), (65, 64, 33, 70, 1.0), (130, 70, 64, 200, 0.37),
    (129, 31, 65, 90, 2.3), (66, 20, 100, 150, 0.6)])
def test_single_view(port, nx, ny, na, ns, ds):
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    g = dict(ns=ns, na=na, ds=ds, orbit=2 * math.pi / na, offset_s=0.3, orbit_start=0.1, nx=nx, ny=ny, dx=1.0, dy=0.9,
             offset_x=0.2, offset_y=-0.3, fov=-1.0)
    op = tc.ParallelBackprojection2DOp(*g.values())
    x = np.random.default_rng(nx).standard_normal((2, na, ns)).astype(np.float32)
    got = host(op.single_view(cuda(x)))
    for b in range(2):
        assert rel_l2(got[b], port.bp_par_2d_sv(x[b], Geom.make(**g))) <= 1e-5
