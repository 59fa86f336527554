"""The border pixels of the FP32 ray-driven adjoint: blocks of 8 pixels of an edge.

Edges shorter than, equal to and just past a block, view counts around the 64
summed side by side, batches with and without a remainder of 4 images: every
border pixel against the oracle, and each image of a batch equal to itself alone.
Reference: src/fp_par_2d.cc:339-383 (one-sided footprints at the image's ends).
"""
import numpy as np
import pytest

from gpu_helpers import cuda, fp_op, host, rel_l2
from test_fp_pairs_gpu import oracle_port  # noqa: F401
from test_fp_plan_gpu import _geom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,na,batch", [
    (1, 5, 2), (2, 3, 1), (3, 64, 4), (7, 1, 5), (8, 63, 2), (9, 65, 1), (16, 130, 9), (17, 90, 3)])
def test_border_pixels(n, na, batch, oracle_port):  # noqa: F811
    from oracle import Geom
    d = _geom(n, na)
    g = Geom.make(**d)
    op = fp_op(d)
    proj = np.random.default_rng(n).standard_normal((batch, na, d["ns"])).astype(np.float32)
    got = host(op.adjoint(cuda(proj)))
    edge = np.ones((n, n), bool)
    edge[1:-1, 1:-1] = False
    for i in range(batch):
        want = oracle_port.fp_par_2d_grad(proj[i], g)
        assert rel_l2(got[i][edge], want[edge]) <= 1e-5
        assert np.array_equal(got[i][edge], host(op.adjoint(cuda(proj[i])))[edge])
