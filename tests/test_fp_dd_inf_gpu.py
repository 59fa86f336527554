"""Infinities and NaN in the sinogram of the FP32 distance-driven grad: each
pixel is the infinity, with its sign, NaN or number that the oracle has, also
where a footprint ends exactly on a channel's (view 0 of the cases that start at
angle 0: the reference then reads a cell of no length).  Finite pixels: the projectors' FP32 bound, rel-L2 1e-5."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ns,ds,offset,start", [(48, 75, 1.0, 0.3, 0.05), (48, 75, 1.0, 0.0, 0.0), (65, 70, 1.3, 0.5, 0.0),
                                                  (40, 130, 0.5, 0.0, 0.0), (70, 300, 0.3, 0.25, -1.0)])
def test_disdriven_grad_infinities(port, n, ns, ds, offset, start):
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    na = 24
    g = dict(ns=ns, na=na, ds=ds, orbit=2 * math.pi / na, offset_s=offset, orbit_start=start, nx=n, ny=n, dx=1.0, dy=1.0,
             offset_x=0.0, offset_y=0.0, fov=-1.0)
    op = tc.ParallelProjection2DOp(*g.values(), method="disdriven")
    rng = np.random.default_rng(ns)
    for value in (np.inf, -np.inf, np.nan, 3.4e38):
        proj = rng.standard_normal((na, ns)).astype(np.float32)
        proj[rng.integers(na if start else 1, size=3), rng.integers(ns, size=3)] = value
        proj[0, ns // 2] = value
        got, want = host(op.adjoint(cuda(proj))), port.fp_par_2d_dd_grad(proj, Geom.make(**g))
        assert np.array_equal(np.isnan(got), np.isnan(want))
        assert np.array_equal(np.isposinf(got), np.isposinf(want)) and np.array_equal(np.isneginf(got), np.isneginf(want))
        fine = np.isfinite(want) & (np.abs(want) < 1e30)
        assert rel_l2(got[fine], want[fine]) <= 1e-5
