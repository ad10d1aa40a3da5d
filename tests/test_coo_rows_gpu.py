"""The row pointer of COO rows: runs of empty rows around the lengths that one thread
fills, at the front, inside and at the end, and products over them."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu
RUN, FAR = 32, 4096   # entries that one thread fills, and its warp


def _rows(case):
    rng = np.random.default_rng(3)
    if case == "none":
        return 1000, np.zeros(0, np.int32)
    if case == "edges":   # runs of RUN - 2 .. RUN + 2 empty rows, and of many
        lens = [x + d for x in (RUN, 256, FAR, 2 * FAR) for d in (-2, -1, 0, 1, 2)] + [9000, 9001]
        at = np.cumsum([x + 1 for x in lens * 3])
        return int(at[-1]) + 1 + RUN, np.repeat(at, rng.integers(1, 40, at.size)).astype(np.int32)
    if case == "front":
        return 100_000, np.full(70, 99_999, np.int32)
    if case == "back":
        return 100_000, np.zeros(70, np.int32)
    if case == "two":
        return 300_000, np.sort(rng.choice([0, 7, 150_000, 299_998], 5000)).astype(np.int32)
    if case == "sparse":
        return 200_000, np.arange(0, 200_000, 1049, dtype=np.int32)
    return 3 * RUN, np.sort(rng.integers(0, 3 * RUN, 9000)).astype(np.int32)


CASES = ["none", "edges", "front", "back", "two", "sparse", "dense"]


@pytest.mark.parametrize("case", CASES)
def test_row_pointer(cuda, case):
    import torch
    nr, rows = _rows(case)
    got = torch.full((nr + 1 + 64,), -7, dtype=torch.int32, device="cuda")
    D.check(D.lib().daspmm_coo_to_csr(nr, rows.size, D._dptr(torch.from_numpy(rows).cuda()),
                                      D._dptr(got), None))
    want = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nr))])
    np.testing.assert_array_equal(got[:nr + 1].cpu().numpy(), want)
    assert (got[nr + 1:] == -7).all()


@pytest.mark.parametrize("case", CASES)
@pytest.mark.parametrize("layout,nv", [(0, 1), (0, 64), (1, 8), (1, 32)])
def test_products(cuda, case, layout, nv):
    import torch
    nr, rows = _rows(case)
    rng = np.random.default_rng(1)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nr))]).astype(np.int32)
    ci = rng.integers(0, 2000, rows.size).astype(np.int32)
    A = D.Csr(nr, 2000, rp, ci, rng.uniform(-1, 1, rows.size).astype(np.float32))
    dA = D.DeviceCsr(A)
    B = D.gen_dense(2000 * nv, seed=nv)
    C0 = D.gen_dense(nr * nv, seed=2)
    c64, absc = O.spmm_f64(layout, nr, 2000, rp, ci, A.values, B, nv)
    for alg in (2, 3):
        C = torch.from_numpy(C0).cuda()
        D.spmm(alg, layout, dA, torch.from_numpy(B).cuda(), C, beta=1.0, nv=nv)
        assert O.rel_err(C.cpu().numpy(), c64 + C0.astype(np.float64),
                         absc + np.abs(C0)) <= O.REL_TOL_F32
