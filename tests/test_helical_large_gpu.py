"""Helical rebinning in FP32 of scans whose output has 2^32 elements and more: the
sample-by-sample kernels with 64-bit indexes, which smaller scans of these shapes
do not take.  Slices of one couch position: each is the one of a scan with a few
(2e-6 of the peak, the bound between the two kernels)."""
import math

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["360", "180"])
def test_output_of_2_to_32(method):
    import torch
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB")
    ns, nt, vpr, nz = 4096, 8, 1024, 1025
    cm = 0.9 * nt * 595.0 / 1085.6 / vpr
    na = 4 * vpr
    x = torch.rand(na, nt, ns, device="cuda", generator=torch.Generator("cuda").manual_seed(3))

    def run(slices):
        op = tc.HelicalInterpolationOp(ns, nt, na, 900.0 / ns, 1.0, 0.375, -0.25, 0.0, 2 * math.pi / vpr, 0.0, cm, vpr, slices,
                                       0.0, (2 * vpr + 3.3) * cm, 1.0, 595.0, 1085.6, method)
        return op.forward(x)

    few = run(2)
    few = few.reshape(-1, vpr, ns)
    peak = float(few.abs().max())
    out = run(nz).reshape(-1, vpr, ns)
    assert out.numel() >= 1 << 32
    for i in (0, 1, 511, 1023, 1024):  # the last from element 2^32 on
        assert float((out[i] - few[0]).abs().max()) <= 2e-6 * peak
