"""The FP32 ramp filter (four rows at a time) against the oracle: rows around the
groups of four, channels around the tasks, the parts and the shared-memory
limits (one row wider than the quad kernels take), launches of few and of many
groups, forward and grad, and a filter with even taps.

Tolerance: the FP32 parity bound (rel-L2 1e-5)."""
import ctypes

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,nrow,batch,kind", [
    (1, 1, 1, 0), (2, 5, 1, 0), (15, 3, 2, 0), (16, 4, 1, 1), (17, 7, 1, 0), (95, 9, 1, 2), (257, 33, 1, 1),
    (300, 50, 30, 0), (769, 6, 1, 0), (1536, 5, 1, 1), (1551, 5, 250, 1), (3100, 3, 1, 0), (4700, 3, 1, 0)])
def test_ramp_rows(port, ns, nrow, batch, kind):
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    op = tc.RampFilterOp(ns, nrow, 0.7, 1085.6, kind)
    x = np.random.default_rng(ns).standard_normal((batch, nrow, ns)).astype(np.float32)
    fwd, adj = host(op.forward(cuda(x))), host(op.adjoint(cuda(x)))
    for b in {0, batch - 1}:
        assert rel_l2(fwd[b], port.ramp_filter(x[b], 0.7, 1085.6, kind)) <= 1e-5
        assert rel_l2(adj[b], port.ramp_filter(x[b], 0.7, 1085.6, kind, grad=True)) <= 1e-5


@pytest.mark.parametrize("ns,nrow", [(40, 6), (700, 9)])
def test_filter_with_even_taps(ns, nrow):
    """Any taps through the C ABI: the plain sum, forward and grad."""
    import torch
    from ct_recon_extensions_gb300 import _lib
    from ct_recon_extensions_gb300.torch_ctrecon import _ptr, _stream
    rng = np.random.default_rng(1)
    h = rng.standard_normal(2 * ns + 1)
    x = rng.standard_normal((nrow, ns)).astype(np.float32)
    p = _lib.FilterParam(ns, nrow, 0.5, -1.0, 0, 0)
    xd, hd = cuda(x), cuda(h)
    out = torch.empty_like(xd)
    i = np.arange(ns)
    T = h[i[:, None] - i[None, :] + ns] * 0.5
    for name, want in (("ctr_ramp_filter_f32", x @ T.T), ("ctr_ramp_filter_grad_f32", x @ T)):
        _lib.call(name, ctypes.byref(p), _ptr(xd), _ptr(hd), _ptr(out), 1, _stream())
        assert rel_l2(host(out), want) <= 1e-5
