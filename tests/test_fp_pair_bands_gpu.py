"""The paired form of the FP32 ray-driven projector on images of 64^2 to 256^2,
in bands of 32 rows: ragged last bands, the smallest paired image and its
unpaired neighbour, even and odd batches.  The same bits image by image, and the
oracle's values (rel-L2 1e-5)."""
import numpy as np
import pytest

from gpu_helpers import cuda, fp_op, host, rel_l2
from test_fp_pairs_gpu import oracle_port  # noqa: F401
from test_fp_plan_gpu import _geom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [62, 64, 66, 80, 100, 130, 254, 256])
@pytest.mark.parametrize("batch", [2, 3, 6])
def test_bands_of_32_rows(n, batch, oracle_port):  # noqa: F811
    import torch
    from oracle import Geom
    d = _geom(n, 13)
    op = fp_op(d)
    imgs = np.random.default_rng(n + batch).standard_normal((batch, n, n)).astype(np.float32)
    imgs[0] = np.nan
    x = cuda(imgs)
    got = op.forward(x)
    for i in range(1, batch):
        assert torch.equal(got[i], op.forward(x[i:i + 1].clone())[0]), i
        assert rel_l2(host(got[i]), oracle_port.fp_par_2d(imgs[i], Geom.make(**d))) <= 1e-5
