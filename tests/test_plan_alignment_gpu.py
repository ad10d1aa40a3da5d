"""Planned products with B and C off the vectors that the plan was made for: widths of
every kernel, offsets of one and two floats, against the FP64 oracle."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 2, 4, 6, 8, 12, 32, 36, 64, 96, 100, 128])
def test_operands_off_their_alignment(cuda, nv):
    import torch
    A = D.gen_powerlaw(6000, seed=nv)
    dA = D.DeviceCsr(A)
    B = D.gen_dense(A.nc * nv, seed=1)
    C0 = D.gen_dense(A.nr * nv, seed=2)
    c64, absc = O.spmm_f64(0, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    plan = D.Plan(dA, nv)
    # the aligned product before, between and after the others
    for off_b, off_c in ((0, 0), (1, 0), (0, 1), (0, 0), (2, 2), (1, 2), (4, 0), (0, 4), (0, 0)):
        for beta in (0.0, 0.5):
            Bt = torch.zeros(B.size + 8, device="cuda")[off_b:off_b + B.size]
            Ct = torch.zeros(C0.size + 8, device="cuda")[off_c:off_c + C0.size]
            Bt.copy_(torch.from_numpy(B))
            Ct.copy_(torch.from_numpy(C0))
            plan.spmm(Bt, Ct, beta=beta)
            assert O.rel_err(Ct.cpu().numpy(), c64 + beta * C0.astype(np.float64),
                             absc + beta * np.abs(C0)) <= O.REL_TOL_F32, (off_b, off_c, beta)


def test_a_vector_the_caller_chose_is_refused(cuda):
    import torch
    A = D.gen_powerlaw(500, seed=1)
    plan = D.Plan(D.DeviceCsr(A), 36, cfg=D.Config(alg=4, vec=4))
    B = torch.zeros(A.nc * 36 + 4, device="cuda")
    C = torch.zeros(A.nr * 36, device="cuda")
    plan.spmm(B, C)
    with pytest.raises(D.DaspmmError):
        plan.spmm(B[1:], C)
