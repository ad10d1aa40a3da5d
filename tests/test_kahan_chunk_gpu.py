"""Rows summed with compensation are cut into pieces of the longest default chunk also in
small products, whose other rows take shorter chunks: every cut adds a rounding that no
compensation covers."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,deg", [(600, 90), (3000, 3)])
@pytest.mark.parametrize("nv,chunk", [(32, 128), (64, 128), (128, 96), (256, 128)])
def test_pieces(cuda, nr, deg, nv, chunk):
    import torch
    A = D.gen_random(nr, 2000, float(deg), seed=nv)
    dA = D.DeviceCsr(A)
    B = D.gen_dense(A.nc * nv, seed=1)
    Bt = torch.from_numpy(B).cuda()
    out = []
    for cfg in (None, D.Config(alg=4, pipe=4, chunk=chunk)):
        C = torch.full((nr * nv,), float("nan"), device="cuda")
        D.spmm_mixed(dA, dA.values, D.Fmt.F32, Bt, D.Fmt.F32, C, nv, kahan_min=1, cfg=cfg)
        out.append(C.cpu().numpy())
    np.testing.assert_array_equal(*out)
    c64, absc = O.spmm_f64(0, nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    # products and sums of a piece are right to a rounding or two, pieces add one each
    pieces = np.repeat(-(-np.diff(A.rowPtr) // chunk) + 1, nv)
    assert (np.abs(out[0] - c64) <= (2 + pieces) * 2.0**-24 * absc).all()
