"""Iso-surfaces through few and through most elements (points formed per
triangle, or for all nodes), against the restatement, bit for bit."""
import numpy as np
import pytest

from oracle import stl as S
from tests import pipeline
from tests.test_gpu_stl import _gpu_case
from tests.test_stl_oracle import _bface_brick

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(pipeline.STL_CASES))
@pytest.mark.parametrize("quantile", [0.002, 0.02, 0.5, 0.999])
def test_sparse_and_dense_surfaces(gpu_lib, name, quantile):
    import torch
    sc, case, g, f, X, x, TMR = _gpu_case(name)
    vals = x[sc["offset"]::sc["vpn"]]
    cut = float(np.quantile(vals, quantile))
    exp = S.triangles(g["oct"], g["conn"], g["dep"], X, x, sc["vpn"], sc["offset"], cut,
                      case["order"], _bface_brick(*sc["grid"]))
    for v in (x, torch.tensor(x, device="cuda")):
        pts = TMR.getSTLTriangles(f, v, offset=sc["offset"], cutoff=cut, vpn=sc["vpn"])
        np.testing.assert_array_equal(pts.reshape(-1, 3, 3), exp)
