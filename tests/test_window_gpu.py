"""The window kernel where it can go wrong: rows without nonzeros (single ones,
runs longer than the rows a worker looks at, at both ends, nearly all rows),
widths and addresses off its vectors, beta, chunks of a few nonzeros, a workspace
without room for the bitmap of empty rows, and an Inf or NaN in the row of B that
pads.  Against the FP64 oracle under its tolerance; rows without nonzeros are
beta*C exactly."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(lens, nc, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(nc, int(k), replace=False)) for k in lens]
                        + [np.zeros(0, int)]).astype(np.int32)
    return D.Csr(len(lens), nc, rp, ci, rng.uniform(-1, 1, int(rp[-1])).astype(np.float32))


def _patterns():
    rng = np.random.default_rng(3)
    single = rng.integers(1, 6, 700)
    single[rng.random(700) < 0.1] = 0
    runs = rng.integers(1, 4, 900)
    for at, n in ((0, 5), (100, 7), (200, 8), (300, 9), (400, 16), (450, 17), (500, 40), (700, 150)):
        runs[at:at + n] = 0
    runs[-33:] = 0
    sparse = np.zeros(5000, int)          # nearly every row is empty
    sparse[rng.choice(5000, 60, replace=False)] = rng.integers(1, 9, 60)
    hubs = rng.integers(0, 3, 500)        # long rows between empty ones
    hubs[[7, 100, 499]] = (900, 333, 64)
    hubs[101:140] = 0
    last = np.zeros(4000, int)            # one nonzero, far down
    last[3999] = 1
    return {"single": single, "runs": runs, "sparse": sparse, "hubs": hubs, "last": last}


@pytest.fixture(scope="module")
def mats(cuda):
    out = {k: _csr(v, 1000, i) for i, (k, v) in enumerate(_patterns().items())}
    return {k: (A, D.DeviceCsr(A)) for k, A in out.items()}


def _product(A, dA, nv, beta, cfg=None, off=0, seed=0, ws=None):
    import torch
    rng = np.random.default_rng(seed)
    B = rng.uniform(-1, 1, A.nc * nv).astype(np.float32)
    C0 = rng.uniform(-1, 1, A.nr * nv).astype(np.float32)
    Bt, Ct = (torch.zeros(x.size + 8, device="cuda")[off:off + x.size] for x in (B, C0))
    Bt.copy_(torch.from_numpy(B))
    Ct.copy_(torch.from_numpy(C0))
    D.spmm(D.Alg.CSR_BALANCED, 0, dA, Bt, Ct, beta=beta, nv=nv, cfg=cfg, workspace=ws)
    return B, C0, Ct.cpu().numpy()


def _check(A, nv, beta, B, C0, C):
    c64, absc = O.spmm_f64(0, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    c64 = c64 + beta * C0.astype(np.float64)
    absc = absc + abs(beta) * np.abs(C0)
    assert O.rel_err(C, c64, absc) <= O.REL_TOL_F32
    none = np.repeat(np.diff(A.rowPtr) == 0, nv)
    np.testing.assert_array_equal(C[none], (np.float32(beta) * C0)[none])


@pytest.mark.parametrize("name", ["single", "runs", "sparse", "hubs", "last"])
@pytest.mark.parametrize("beta", [0.0, 0.5, 1.0])
def test_empty_rows(mats, name, beta):
    A, dA = mats[name]
    for nv in (17, 18, 20, 32, 33, 41, 48, 50, 64, 66, 96, 100, 101, 128, 129, 200, 256):
        for kw in ({}, dict(chunk=7, snap=3), dict(chunk=40)):
            cfg = D.Config(alg=int(D.Alg.CSR_BALANCED), **kw)
            _check(A, nv, beta, *_product(A, dA, nv, beta, cfg))


@pytest.mark.parametrize("off", [1, 2, 3, 4])
def test_alignment(mats, off):
    for name in ("single", "hubs"):
        A, dA = mats[name]
        for nv in (18, 20, 41, 64, 66, 96, 100, 128, 130, 256):
            for beta in (0.0, 0.5):
                _check(A, nv, beta, *_product(A, dA, nv, beta, off=off))


@pytest.mark.parametrize("nv", [32, 41, 64, 100, 128, 256])
def test_without_the_bitmap(mats, nv):
    """The least workspace has no room for the bitmap: the same bits."""
    import torch
    for name in ("single", "runs", "hubs"):
        A, dA = mats[name]
        cfg = D.default_config(D.Alg.CSR_BALANCED, 0, A.nr, A.nc, A.nnz, nv)
        full = D.workspace_bytes(cfg, 0, A.nr, A.nc, A.nnz, nv)
        bitmap = ((A.nr + 31) // 32 * 4 + 255) // 256 * 256
        got = [_product(A, dA, nv, 0.0, cfg, ws=torch.empty(n, dtype=torch.uint8, device="cuda"))[2]
               for n in (full, full - bitmap)]
        np.testing.assert_array_equal(*got)


@pytest.mark.parametrize("vf,bf", [(1, 1), (2, 2), (0, 3), (1, 3)])
def test_reduced_precision(mats, vf, bf):
    """Empty rows and beta with reduced storage: the aligned shapes and those for C
    off their alignment give the same bits, and the product of the stored values."""
    import torch
    for name in ("single", "runs", "hubs"):
        A, dA = mats[name]
        vq = D.quantize(dA.values, vf) if vf else dA.values
        for nv in (32, 64, 128, 256):
            B = torch.rand(A.nc * nv, device="cuda") * 2 - 1
            sc = D.e4m3_scales(B, A.nc, nv) if bf == 3 else None
            bq = D.quantize(B, bf, sc, nv if bf == 3 else 0)
            C0 = torch.rand(A.nr * nv, device="cuda")
            for beta in (0.0, 0.5):
                Ca = C0.clone()
                Co = torch.zeros(A.nr * nv + 8, device="cuda")[4:4 + A.nr * nv]
                Co.copy_(C0)
                for C in (Ca, Co):
                    D.spmm_mixed(dA, vq, vf, bq, bf, C, nv, b_scales=sc, beta=beta)
                assert torch.equal(Ca, Co)
                v64 = (vq.double() if vf else dA.values.double()).cpu().numpy()
                b64 = (bq.view(torch.float8_e4m3fn).double().view(A.nc, nv) * sc.double()
                       if bf == 3 else bq.double()).cpu().numpy().reshape(-1)
                c64, absc = O.spmm_f64d(0, A.nr, A.nc, A.rowPtr, A.colIdx, v64, b64, nv)
                old = C0.double().cpu().numpy()
                assert O.rel_err(Ca.cpu().numpy(), c64 + beta * old,
                                 absc + beta * np.abs(old)) <= O.REL_TOL_F32


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("nv", [32, 41, 64, 100, 128, 256])
def test_padding_row_not_finite(mats, bad, nv):
    """Row 0 of B, which short windows pad with, is not finite: what is not finite in
    C is what the host loop has so, with rows that use row 0 and without."""
    import torch
    for name in ("single", "hubs"):
        for shift in (0, 1):
            A0 = mats[name][0]
            A = D.Csr(A0.nr, A0.nc + 1, A0.rowPtr, A0.colIdx + shift, A0.values)
            dA = D.DeviceCsr(A)
            B = np.random.default_rng(1).uniform(-1, 1, A.nc * nv).astype(np.float32)
            B[:nv:3] = bad
            want = O.spmm_f32(0, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
            for chunk in (0, 7):
                C = torch.full((A.nr * nv,), 7.0, device="cuda")
                D.spmm(D.Alg.CSR_BALANCED, 0, dA, torch.from_numpy(B).cuda(), C, nv=nv,
                       cfg=D.Config(alg=4, chunk=chunk))
                got = C.cpu().numpy()
                fine = np.isfinite(want)
                np.testing.assert_array_equal(np.isfinite(got), fine)
                np.testing.assert_array_equal(got[~fine], want[~fine])
                assert np.abs(got[fine] - want[fine]).max() <= O.REF_ABS_TOL

