"""Ray casting by image rows (steps up to half a pixel) against the oracle: image
sides around the copies' tiles and the detector chunks, non-square images, rays
along the axes and the diagonals, steps around the rule's limit.

Tolerance: the FP32 parity bound of the projectors (rel-L2 1e-5)."""
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ns,na,step,start", [
    (1, 1, 5, 4, 0.5, 0.1), (28, 28, 127, 8, 0.125, 0.0), (29, 60, 128, 9, 0.25, math.pi / 4),
    (61, 28, 129, 12, 0.01, 0.3), (33, 92, 257, 16, 0.5, 0.0), (92, 33, 50, 16, 0.51, 0.0),
    (64, 64, 65, 10, 0.37, 0.7), (31, 31, 64, 7, 1.0, 0.0),
    (40, 40, 64, 7, 3.0, 0.2),
    # enough samples for the rows
    (1, 1, 31, 1700, 0.1, 0.1), (28, 28, 127, 20, 0.125, 0.0), (29, 60, 128, 36, 0.25, math.pi / 4),
    (33, 92, 257, 32, 0.5, 0.0), (92, 33, 50, 160, 0.5, 0.0), (64, 64, 65, 48, 0.37, 0.7), (30, 30, 33, 130, 0.25, 0.2)])
def test_cast_rows(port, nx, ny, ns, na, step, start):
    from oracle import Geom
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    orbit = 2 * math.pi / na  # all directions, both signs of both steps
    args = dict(ns=ns, na=na, ds=0.8 * max(nx, ny) / ns + 0.1, orbit=orbit, offset_s=0.3, orbit_start=start, nx=nx,
                ny=ny, dx=1.0, dy=0.8, offset_x=0.25, offset_y=-0.6, fov=0.45 * (nx + ny) + 2.0)
    op = tc.ParallelProjection2DOp(*args.values(), method="raycasting", step_size=step)
    img = np.random.default_rng(nx + ns).random((2, ny, nx)).astype(np.float32)
    out = host(op.forward(cuda(img)))
    for b in range(2):
        assert rel_l2(out[b], port.fp_par_2d_cast(img[b], Geom.make(**args), step)) <= 1e-5
        assert np.array_equal(out[b], host(op.forward(cuda(img[b]))))
