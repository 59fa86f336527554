"""The FP32 fan weighting equals the FP64 product rounded to float, bit for bit:
weights from the FP64 operator (of ones), inputs over the whole range of float,
midpoints of two floats, zeros, denormals, infinities and NaN, in place, sizes
around a CTA's channels and rows."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import cuda, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nrow,batch,kind", [(1, 1, 1, 1), (31, 7, 1, 1), (33, 31, 2, 2), (64, 33, 3, 1), (700, 129, 1, 1),
                                                (95, 2000, 4, 2)])
def test_rounds_the_fp64_product(ns, nrow, batch, kind):
    import torch
    from ct_recon_extensions_gb300 import _lib
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    op = tc.FanWeightingOp(ns, nrow, 1.3, 0.25, 595.0, 1085.6, kind)
    rng = np.random.default_rng(ns)
    x = (rng.standard_normal((batch, nrow, ns)) * 10.0 ** rng.uniform(-44, 38, (batch, nrow, ns))).astype(np.float32)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-45, -1e-40, 3.4e38, 1.0], np.float32)
    put = rng.random(x.shape) < 0.2
    x[put] = rng.choice(special, put.sum())
    w = host(op.forward(torch.ones((nrow, ns), dtype=torch.float64, device="cuda")))
    # products next to the midpoint of two floats
    m = (rng.integers(1 << 23, 1 << 24, x.shape) + 0.5) / 2 ** 24
    near = rng.random(x.shape) < 0.2
    x[near] = (m / w)[near].astype(np.float32)
    with np.errstate(all="ignore"):
        want = (w * x.astype(np.float64)).astype(np.float32)
    for got in (host(op.forward(cuda(x))), host(op.adjoint(cuda(x)))):
        assert np.array_equal(got.view(np.uint32)[~np.isnan(want)], want.view(np.uint32)[~np.isnan(want)])
        assert np.isnan(got[np.isnan(want)]).all()
    y = cuda(x)
    _lib.call("ctr_fan_weighting_f32", ctypes.byref(op.p), tc._ptr(y), tc._ptr(y), batch, tc._stream())
    assert np.array_equal(host(y), got, equal_nan=True)
