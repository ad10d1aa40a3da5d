"""Column-major balanced CSR through a row-major product: its two transposes at
the edges of their tiles (every tile shape, vector and single accesses on either
side) move values, so the product is bit for bit the row-major one."""
import numpy as np
import pytest

import daspmm as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 255, 257, 1000])
@pytest.mark.parametrize("nv", [4, 5, 16, 17, 32, 33, 63, 64, 65, 100, 128])
@pytest.mark.parametrize("off", [0, 1])
@pytest.mark.parametrize("beta", [0.0, 0.5])
def test_equals_row_major(cuda, rows, nv, off, beta):
    import torch
    A = D.gen_random(rows, rows + 3, 3.0, seed=rows)
    dA = D.DeviceCsr(A)
    g = torch.Generator("cuda").manual_seed(rows * nv)
    B = torch.rand(A.nc, nv, generator=g, device="cuda")
    C0 = torch.rand(A.nr, nv, generator=g, device="cuda")
    want = torch.empty(A.nr, nv, device="cuda")
    D.spmm(D.Alg.CSR_BALANCED, 0, dA, B, want, nv=nv)
    Bc = torch.empty(A.nc * nv + off, device="cuda")[off:]
    Cc = torch.empty(A.nr * nv + off, device="cuda")[off:]
    Bc.copy_(B.t().reshape(-1))
    Cc.copy_(C0.t().reshape(-1))
    D.spmm(D.Alg.CSR_BALANCED, 1, dA, Bc, Cc, beta=beta, nv=nv,
           cfg=D.Config(alg=int(D.Alg.CSR_BALANCED), pipe=5))
    got = Cc.view(nv, A.nr).t()
    if beta:  # one more rounding: fma(beta, C0, sum)
        want = (want.double() + beta * C0.double()).float()
        assert torch.equal(got, want)
    else:
        assert torch.equal(got, want)
