"""The FP32 ray-driven projector on batches: pairs of images, the odd one left.

A ray's value does not depend on the batch it is in: image by image, pairs, and
pairs with one image over give the same bits, through the per-call entry point
and a plan, and match the oracle.  Sizes: one and two bands of 16 rows, a ragged
last band, the largest paired image (512) and the unpaired ones (odd, 514); a
neighbour full of NaN does not reach the other image of its pair.
Reference: src/fp_par_2d.cc:149-280.
"""
import numpy as np
import pytest

from gpu_helpers import cuda, fp_op, host, rel_l2
from test_fp_plan_gpu import _geom, _per_call, _plan

pytestmark = pytest.mark.gpu

TOL = 1e-5  # the projector's bound against the oracle at every size


@pytest.fixture(scope="module")
def oracle_port():
    import os
    from oracle import Oracle
    return Oracle("port", threads=os.cpu_count() or 1)


@pytest.mark.parametrize("n,na,batch", [
    (2, 5, 2), (16, 9, 3), (30, 8, 2), (33, 7, 4), (256, 12, 3), (258, 11, 5), (272, 10, 2), (510, 9, 3),
    (512, 21, 4), (514, 6, 3)])
def test_pairs_match_single_images(n, na, batch, oracle_port):
    import torch
    from oracle import Geom
    d = _geom(n, na)
    g = Geom.make(**d)
    op = fp_op(d)
    imgs = np.random.default_rng(n).standard_normal((batch, n, n)).astype(np.float32)
    imgs[0] = np.nan
    x = cuda(imgs)
    tables = op.tables(torch.device("cuda"))
    got = _per_call(op, x, tables)
    planned = _plan(op, x, tables, (batch,))[0]
    assert torch.equal(got[1:], planned[1:])
    for i in range(1, batch):
        assert torch.equal(got[i:i + 1], _per_call(op, x[i:i + 1].clone(), tables)), i
        assert rel_l2(host(got[i]), oracle_port.fp_par_2d(imgs[i], g)) <= TOL
