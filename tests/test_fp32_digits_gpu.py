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
