"""The FP32 ray-driven adjoint's view segments: partial images or launches in turn.

One image of these sizes takes every segment at once (partial images), the batch a
launch a segment, each adding to the one before it: the same bits, the oracle's
values, and the same again from a captured graph.  View counts: fewer views than
segments of 16, one over a multiple, several segments each.
Reference: src/fp_par_2d.cc:285-391.
"""
import numpy as np
import pytest

from gpu_helpers import cuda, fp_op, host, rel_l2
from test_fp_pairs_gpu import oracle_port  # noqa: F401
from test_fp_plan_gpu import _geom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,na,batch", [(64, 33, 160), (200, 129, 24), (512, 17, 5), (512, 145, 3), (640, 100, 2)])
def test_segments_in_turn_match_partial_images(n, na, batch, oracle_port):  # noqa: F811
    import torch
    from oracle import Geom
    d = _geom(n, na)
    op = fp_op(d)
    proj = np.random.default_rng(n + na).standard_normal((batch, na, d["ns"])).astype(np.float32)
    x = cuda(proj)
    got = op.adjoint(x)
    for i in (0, batch // 2, batch - 1):
        assert torch.equal(got[i], op.adjoint(x[i].clone())), i
    assert rel_l2(host(got[-1]), oracle_port.fp_par_2d_grad(proj[-1], Geom.make(**d))) <= 1e-5
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = op.adjoint(x)
    for _ in range(2):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, got)
