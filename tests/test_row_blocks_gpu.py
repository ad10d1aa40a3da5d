"""Rows of a larger matrix: the CSR algorithms and AUTO take rowPtr + r with the whole
matrix's colIdx and values, whatever nnz of the two they are given, in their own kernels
and as the balanced product."""
import copy

import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mat(cuda):
    rng = np.random.default_rng(4)
    n = 230_000
    lens = np.minimum((rng.pareto(1.1, n) * 3).astype(int), 3000)
    lens[rng.random(n) < 0.1] = 0
    lens[100_000:120_000] = 0            # a run of empty rows
    lens[[80_000, 149_999, 150_000]] = 900
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = rng.integers(0, 5000, int(rp[-1])).astype(np.int32)
    A = D.Csr(n, 5000, rp, ci, rng.uniform(-1, 1, int(rp[-1])).astype(np.float32))
    return A, D.DeviceCsr(A)


# (first row, last row): from the front, the middle, to the end, inside the empty run
BLOCKS = [(0, 80_001), (79_000, 150_000), (150_000, 230_000), (101_000, 119_000), (229_990, 230_000)]


@pytest.mark.parametrize("r0,r1", BLOCKS)
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nv", [1, 4, 8, 16, 41, 128])
def test_row_block(mat, r0, r1, layout, nv):
    import torch
    D.lib().daspmm_tune_clear()
    A, dA = mat
    part = copy.copy(dA)
    part.nr, part.rowPtr = r1 - r0, dA.rowPtr[r0:r1 + 1]
    k0, k1 = int(A.rowPtr[r0]), int(A.rowPtr[r1])
    B = D.gen_dense(A.nc * nv, seed=nv)
    C0 = D.gen_dense(part.nr * nv, seed=2)
    Bt = torch.from_numpy(B).cuda()
    c64, absc = O.spmm_f64(layout, part.nr, A.nc, (A.rowPtr[r0:r1 + 1] - k0).astype(np.int32),
                           A.colIdx[k0:k1].copy(), A.values[k0:k1].copy(), B, nv)
    for nnz in (k1 - k0, A.nnz):
        part.nnz = nnz
        for alg in (0, 1, 5):
            if alg == 5 and layout == 0 and nv >= 32:
                continue   # AUTO's configuration is the balanced product, which needs its own nnz
            for beta in (0.0, 0.5):
                C = torch.from_numpy(C0).cuda()
                D.spmm(alg, layout, part, Bt, C, beta=beta, nv=nv)
                assert O.rel_err(C.cpu().numpy(), c64 + beta * C0.astype(np.float64),
                                 absc + beta * np.abs(C0)) <= O.REL_TOL_F32, (nnz, alg, beta)
