"""Products of few columns over matrices with far more rows than nonzeros, or with their
empty rows in one place: chunks of more rows than one CTA walks, with rows cut at their
boundaries, in both layouts and with every kind of beta."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu
LIMIT = 4096   # rows between two boundaries that one CTA walks


def _csr(lens, seed):
    rng = np.random.default_rng(seed)
    nc = 3000
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = [np.sort(rng.choice(nc, int(k), replace=False)) for k in lens if k]
    ci = np.concatenate(ci + [np.zeros(0, int)]).astype(np.int32)
    return D.Csr(len(lens), nc, rp, ci, rng.uniform(-1, 1, int(rp[-1])).astype(np.float32))


def _matrices():
    rng = np.random.default_rng(7)
    runs = []
    # rows that are cut on both sides of a run of empty rows, short and long rows inside
    for k, run in enumerate((LIMIT - 2, LIMIT - 1, LIMIT, LIMIT + 1, 9000, 40_000)):
        gap = np.zeros(run, int)
        gap[rng.choice(run, 12, replace=False)] = rng.choice([1, 2, 16, 17, 40, 96, 130], 12)
        runs += [[300 + 64 * k], gap, rng.integers(0, 5, 50)]
    half = np.concatenate([rng.integers(0, 6, 3000), np.zeros(70_000, int)])
    sparse = np.zeros(120_000, int)
    sparse[::977] = 1
    last = np.zeros(20_000, int)
    last[-1] = 700
    first = last[::-1].copy()
    out = {"runs": np.concatenate(runs), "runs_back": np.concatenate(runs)[::-1], "half": half,
           "half_back": half[::-1], "sparse": sparse, "last": last, "first": first,
           "none": np.zeros(10_000, int), "one": np.eye(1, 9000, 4500, dtype=int)[0]}
    return {k: _csr(v, i) for i, (k, v) in enumerate(out.items())}


@pytest.fixture(scope="module")
def mats(cuda):
    return {k: (A, D.DeviceCsr(A)) for k, A in _matrices().items()}


@pytest.mark.parametrize("name", ["runs", "runs_back", "half", "half_back", "sparse", "last",
                                  "first", "none", "one"])
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nv", [1, 2, 3, 4, 7, 8])
def test_rows_of_a_long_run(mats, name, layout, nv):
    import torch
    A, dA = mats[name]
    B = D.gen_dense(A.nc * nv, seed=nv)
    C0 = D.gen_dense(A.nr * nv, seed=9)
    Bt = torch.from_numpy(B).cuda()
    c64, absc = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    empty = np.diff(A.rowPtr) == 0
    for beta in (0.0, 0.5, 1.0):
        C = torch.from_numpy(C0 if beta else np.full_like(C0, np.nan)).cuda()
        for cfg in (None, D.Config(alg=4, chunk=256)):
            Ct = C.clone()
            D.spmm(4, layout, dA, Bt, Ct, beta=beta, nv=nv, cfg=cfg)
            got = Ct.cpu().numpy()
            assert O.rel_err(got, c64 + beta * C0.astype(np.float64),
                             absc + beta * np.abs(C0)) <= O.REL_TOL_F32
            if beta == 1.0:
                rows = (x.reshape(A.nr, nv) if layout == 0 else x.reshape(nv, A.nr).T
                        for x in (got, C0))
                np.testing.assert_array_equal(*(r[empty] for r in rows))


def test_a_workspace_that_holds_anything(mats):
    """What says that rows were left is never cleared: whatever the memory holds is right."""
    import torch
    for name in ("half", "runs"):
        A, dA = mats[name]
        B = D.gen_dense(A.nc * 4, seed=4)
        Bt = torch.from_numpy(B).cuda()
        c64, absc = O.spmm_f64(0, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, 4)
        cfg = D.Config(alg=4)
        for fill in (0, 1, 255):
            ws = torch.full((D.workspace_bytes(cfg, 0, A.nr, A.nc, A.nnz, 4),), fill,
                            dtype=torch.uint8, device="cuda")
            C = torch.full((A.nr * 4,), float("nan"), device="cuda")
            for _ in range(3):
                D.spmm(4, 0, dA, Bt, C, nv=4, cfg=cfg, workspace=ws)
                assert O.rel_err(C.cpu().numpy(), c64, absc) <= O.REL_TOL_F32
