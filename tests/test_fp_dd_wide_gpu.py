"""The FP32 distance-driven grad with pixels long one way and flat the other, as
wide as the tiles' windows of channels take (the host rule's edge) and beyond,
against the oracle: rel-L2 within 1e-5, the projectors' FP32 bound."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dx,dy", [(3.5, 0.2), (3.5, 0.1), (3.0, 0.9), (3.0, 0.95), (0.2, 1.75), (0.1, 1.8), (3.6, 0.2)])
def test_disdriven_grad_long_pixels(port, dx, dy):
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    n, na, ns = 70, 34, 330
    g = dict(ns=ns, na=na, ds=1.0, orbit=2 * math.pi / na, offset_s=0.3, orbit_start=0.0, nx=n, ny=n, dx=dx, dy=dy,
             offset_x=0.25, offset_y=-0.6, fov=-1.0)
    proj = np.random.default_rng(n).standard_normal((na, ns)).astype(np.float32)
    got = host(tc.ParallelProjection2DOp(*g.values(), method="disdriven").adjoint(cuda(proj)))
    assert rel_l2(got, port.fp_par_2d_dd_grad(proj, Geom.make(**g))) <= 1e-5
