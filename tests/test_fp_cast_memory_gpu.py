"""The memory of FP32 ray casting by rows: none of the device's default pool
unless the C entry without scratch has enough to do; as many images at a time as
fit, each with the same result; under capture; without memory sample by sample."""
import ctypes
import math

import numpy as np
import pytest

from gpu_helpers import cuda, host, rel_l2
from test_zz_no_alloc import _cudart

pytestmark = pytest.mark.gpu


def _op(n, na, ns, step):
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    return tc.ParallelProjection2DOp(ns, na, 1.0, math.pi / na, 0.25, 0.1, n, n, 1.0, 1.0, 0.0, 0.0, fov=0.45 * n,
                                     method="raycasting", step_size=step)


def _plain(op, x):
    """ctr_fp_par_2d_cast_f32."""
    import torch
    from ct_recon_extensions_gb300._lib import call
    from ct_recon_extensions_gb300.torch_ctrecon import _ptr, _stream
    out = torch.empty((x.shape[0], op.na, op.ns), dtype=torch.float32, device=x.device)
    call("ctr_fp_par_2d_cast_f32", ctypes.byref(op.p), op.step_size, _ptr(x), _ptr(out), *map(_ptr, op.tables(x.device)),
         x.shape[0], _stream())
    return out


def _pool_growth(f):
    import torch
    rt, pool = _cudart(), ctypes.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    torch.cuda.synchronize()
    zero, now, high = ctypes.c_uint64(0), ctypes.c_uint64(), ctypes.c_uint64()
    assert rt.cudaMemPoolSetAttribute(pool, 8, ctypes.byref(zero)) == 0
    assert rt.cudaMemPoolGetAttribute(pool, 7, ctypes.byref(now)) == 0
    f()
    torch.cuda.synchronize()
    assert rt.cudaMemPoolGetAttribute(pool, 8, ctypes.byref(high)) == 0
    return high.value - now.value


def test_default_pool():
    import torch
    small, large = _op(114, 152, 165, 0.5), _op(300, 300, 430, 0.125)
    xs, xl = cuda(np.ones((2, 114, 114), np.float32)), cuda(np.random.default_rng(1).random((2, 300, 300)).astype(np.float32))
    assert small._lib.ctr_fp_par_2d_cast_scratch(ctypes.byref(small.p), 0.5) == 2 * 4 * 118 ** 2
    for op, x in ((small, xs), (large, xl)):
        op.forward(x)
        assert _pool_growth(lambda: op.forward(x)) == 0
    assert _pool_growth(lambda: _plain(small, xs)) == 0  # sample by sample
    assert _pool_growth(lambda: _plain(large, xl)) > 0
    assert torch.equal(_plain(large, xl), large.forward(xl))
    assert rel_l2(host(_plain(small, xs)), host(small.forward(xs))) <= 1e-6


def test_images_at_a_time(monkeypatch):
    import torch
    from ct_recon_extensions_gb300 import torch_ctrecon as tc
    op = _op(90, 100, 130, 0.25)
    x = cuda(np.random.default_rng(2).random((7, 90, 90)).astype(np.float32))
    want = op.forward(x)
    one = op._lib.ctr_fp_par_2d_cast_scratch(ctypes.byref(op.p), 0.25)
    for most in (1, 3 * one + 5, 7 * one):
        monkeypatch.setattr(tc, "_CAST_BYTES", most)
        assert torch.equal(op.forward(x), want)
    # no room for more than two images', then for none: the same, then sample by sample
    empty = torch.empty
    for room in (2, 0):
        def short(*a, **kw):
            if kw.get("dtype") == torch.uint8 and a[0] > room * one:
                raise torch.cuda.OutOfMemoryError("no room")
            return empty(*a, **kw)
        monkeypatch.setattr(torch, "empty", short)
        got = op.forward(x)
        monkeypatch.setattr(torch, "empty", empty)
        assert torch.equal(got, want) if room else rel_l2(host(got), host(want)) <= 1e-6 and not torch.equal(got, want)


def test_capture():
    import torch
    op = _op(90, 100, 130, 0.25)
    x = cuda(np.random.default_rng(3).random((2, 90, 90)).astype(np.float32))
    want = op.forward(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = op.forward(x)
    x2 = x.clone()
    x.mul_(2)
    g.replay()
    assert torch.equal(out, op.forward(x)) and torch.equal(op.forward(x2), want)


def test_scratch_refused():
    from ct_recon_extensions_gb300 import _lib
    lib = _lib.load()
    p = _op(90, 100, 130, 0.25).p
    assert lib.ctr_fp_par_2d_cast_f32_scratch(ctypes.byref(p), 0.25, 1, 2, 3, 4, 5, 1, None, 100, None) == 1
    assert lib.ctr_fp_par_2d_cast_f32_scratch(ctypes.byref(p), 0.25, 1, 2, 3, 4, 5, 1, 6, 100, None) == 1
