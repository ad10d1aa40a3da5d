"""beta == 1 leaves the rows of C that have no nonzeros alone: a -0.0 there (which
1 * C + 0 would make +0.0) stays, and calls on disjoint rows of one C may overlap."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _half(nr, which, seed):
    """Rows of two halves that take turns in runs of 1 to 700 rows; the others are empty."""
    rng = np.random.default_rng(seed)
    cuts = np.cumsum(np.random.default_rng(9).integers(1, 700, nr))
    mine = (np.searchsorted(cuts, np.arange(nr), side="right") % 2) == which
    lens = np.where(mine, rng.integers(1, 12, nr), 0)
    lens[np.flatnonzero(mine)[[0, 5, -1]]] = (300, 900, 130)   # rows that are cut
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(nr, int(k), replace=False)) if k > 64
                         else (int(rng.integers(nr - 64)) + np.arange(k)) for k in lens if k])
    va = rng.uniform(-1, 1, int(rp[-1])).astype(np.float32)
    return D.Csr(nr, nr, rp, ci.astype(np.int32), va), mine


@pytest.fixture(scope="module", params=[30_001, 30_004])   # rows off and on four
def halves(cuda, request):
    out = [_half(request.param, w, w) for w in (0, 1)]
    assert not (out[0][1] & out[1][1]).any()
    return [(A, D.DeviceCsr(A), mine) for A, mine in out]


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nv", [1, 2, 4, 7, 8, 16, 32, 41, 128])
def test_rows_without_nonzeros(halves, layout, nv):
    import torch
    A, dA, mine = halves[0]
    nr = A.nr
    B = D.gen_dense(nr * nv, seed=1)
    Bt = torch.from_numpy(B).cuda()
    c64, absc = O.spmm_f64(layout, nr, nr, A.rowPtr, A.colIdx, A.values, B, nv)
    C0 = np.full((nr, nv) if layout == 0 else (nv, nr), -0.0, np.float32)
    (C0 if layout == 0 else C0.T)[mine] = 2.0
    for alg in range(6):
        C = torch.from_numpy(C0.reshape(-1).copy()).cuda()
        D.spmm(alg, layout, dA, Bt, C, beta=1.0, nv=nv)
        got = C.cpu().numpy()
        assert O.rel_err(got, c64 + C0.reshape(-1).astype(np.float64),
                         absc + np.abs(C0.reshape(-1))) <= O.REL_TOL_F32
        if alg in (2, 3, 4):   # (CSR scalar and vector write every row)
            rows = got.reshape(C0.shape) if layout == 0 else got.reshape(C0.shape).T
            assert np.signbit(rows[~mine]).all(), alg


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("alg", [D.Alg.COO_SCALAR, D.Alg.COO_VECTOR])
@pytest.mark.parametrize("nv", [4, 64])
def test_two_streams_add_into_one(halves, alg, layout, nv):
    import torch
    nr = halves[0][0].nr
    B = D.gen_dense(nr * nv, seed=1)
    Bt = torch.from_numpy(B).cuda()
    C = torch.zeros(nr * nv, device="cuda")
    streams = [torch.cuda.Stream() for _ in halves]
    torch.cuda.synchronize()
    times = 40
    for _ in range(times):
        for (A, dA, _), st in zip(halves, streams):
            D.spmm(alg, layout, dA, Bt, C, beta=1.0, nv=nv, stream=st)
    torch.cuda.synchronize()
    want, absw = 0.0, 0.0
    for A, _, _ in halves:
        c64, absc = O.spmm_f64(layout, nr, nr, A.rowPtr, A.colIdx, A.values, B, nv)
        want, absw = want + times * c64, absw + times * absc
    assert O.rel_err(C.cpu().numpy(), want, absw) <= O.REL_TOL_F32
