"""Distance-driven calls with next to no device memory left: the C entries' own
scratch does not fit for all images, or for any, and the calls still give their
results (fewer images at a time: the same ones)."""
import ctypes
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu


class _Left:
    """At most `mib` MiB of the device's memory left while it is held."""

    def __init__(self, mib):
        self.left = mib << 20

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.held = []
        size = 1 << 36
        while size >= 1 << 23:
            if torch.cuda.mem_get_info()[0] - self.left >= size:
                try:
                    self.held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
                    continue
                except torch.cuda.OutOfMemoryError:
                    pass
            size //= 2

    def __exit__(self, *a):
        import torch
        torch.cuda.synchronize()
        self.held.clear()
        torch.cuda.empty_cache()


def _op(n, na, ns, **kw):
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    return tc.ParallelProjection2DOp(ns, na, n / ns, math.pi / na, 0.25, 0.1, n, n, 1.0, 1.0, 0.0, 0.0, **kw)


@pytest.mark.parametrize("mib", [110, 48])
def test_disdriven_forward(mib):
    """Two images of 3000^2 (72 MB of copies each): one at a time, then ray by ray
    (sums and divisions per line against scaled sums: 1e-6)."""
    import torch
    op = _op(3000, 6, 700, method="disdriven")
    x = torch.rand(2, 3000, 3000, device="cuda")
    want = op.forward(x)
    out = torch.empty_like(want)
    from ct_recon_extensions_gb300._lib import call
    from ct_recon_extensions_gb300.torch_ctrecon import _ptr, _stream
    with _Left(mib):
        call("ctr_fp_par_2d_dd_f32", ctypes.byref(op.p), _ptr(x), _ptr(out), *map(_ptr, op.tables(x.device)), 2, _stream())
        torch.cuda.synchronize()
    if mib == 110:
        assert torch.equal(out, want)
    assert rel_l2(host(out), host(want)) <= 1e-6


@pytest.mark.parametrize("mib", [200, 48])
def test_disdriven_grad(mib):
    """Six images of 1100^2 with partial images of 16 segments (77 MB each): fewer at
    a time, then none (other sums of the same 64 terms a pixel: 1e-6). """
    import torch
    op = _op(1100, 512, 150, method="disdriven")
    x = torch.randn(6, 512, 150, device="cuda")
    want = op.adjoint(x)
    out = torch.empty_like(want)
    from ct_recon_extensions_gb300._lib import call
    from ct_recon_extensions_gb300.torch_ctrecon import _ptr, _stream
    tables = op.grad_tables(x.device)
    with _Left(mib):
        call("ctr_fp_par_2d_dd_grad_f32", ctypes.byref(op.p), _ptr(x), _ptr(out), *map(_ptr, tables), 6, _stream())
        torch.cuda.synchronize()
    if mib == 200:
        assert torch.equal(out, want)
    assert rel_l2(host(out), host(want)) <= 1e-6


def test_disdriven_grad_many_images():
    """More images than a grid takes with their segments: each as by itself."""
    import torch
    op = _op(8, 300, 12, method="disdriven")
    x = torch.randn(9000, 300, 12, device="cuda")
    got = op.adjoint(x)
    for i in (0, 4095, 6552, 6553, 8999):
        assert torch.equal(got[i], op.adjoint(x[i]))
