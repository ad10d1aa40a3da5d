"""Products of few columns (k_stream) and the reference's algorithms run as the
balanced product: chunk and row boundaries, rows cut once and many times, empty
rows, both layouts, beta, addresses off the vectors, non-finite operands, and the
calls that keep their own kernels (stream capture, no room for the workspace)."""
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


@pytest.fixture(scope="module")
def mats(cuda):
    rng = np.random.default_rng(2)
    short = rng.integers(0, 9, 3000)
    cut = rng.integers(0, 4, 400)                 # rows around the lengths that are cut or
    cut[::7] = rng.choice([62, 63, 64, 65, 95, 96, 97, 127, 128, 129, 200], cut[::7].size)
    hub = rng.integers(0, 3, 300)
    hub[[0, 150, 299]] = (5000, 1500, 700)        # over many chunks, first and last row too
    empty = np.zeros(4000, int)
    empty[[17, 2000, 3998]] = (1, 700, 3)
    out = {"short": _csr(short, 900, 1), "cut": _csr(cut, 900, 2), "hub": _csr(hub, 6000, 3),
           "empty": _csr(empty, 900, 4), "one": _csr([1], 1, 5)}
    return {k: (A, D.DeviceCsr(A)) for k, A in out.items()}


def _run(A, dA, alg, layout, nv, beta, off=0, cfg=None, bad=None):
    import torch
    rng = np.random.default_rng(nv)
    B = rng.uniform(-1, 1, A.nc * nv).astype(np.float32)
    if bad is not None:
        B[:: 2 * nv + 1] = bad
    C0 = rng.uniform(-1, 1, A.nr * nv).astype(np.float32)
    Bt, Ct = (torch.zeros(x.size + 8, device="cuda")[off:off + x.size] for x in (B, C0))
    Bt.copy_(torch.from_numpy(B))
    Ct.copy_(torch.from_numpy(C0))
    D.spmm(alg, layout, dA, Bt, Ct, beta=beta, nv=nv, cfg=cfg)
    return B, C0, Ct.cpu().numpy()


def _check(A, layout, nv, beta, B, C0, C):
    c64, absc = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    assert O.rel_err(C, c64 + beta * C0.astype(np.float64),
                     absc + abs(beta) * np.abs(C0)) <= O.REL_TOL_F32


@pytest.mark.parametrize("name", ["short", "cut", "hub", "empty", "one"])
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nv", [1, 2, 3, 4, 5, 6, 7, 8, 9, 12, 16])
def test_few_columns(mats, name, layout, nv):
    A, dA = mats[name]
    for beta in (0.0, 0.5):
        for off in (0, 1, 2):
            _check(A, layout, nv, beta, *_run(A, dA, 4, layout, nv, beta, off))
    for chunk in (128, 256):   # an explicit chunk of the same kernel
        _check(A, layout, nv, 0.0,
               *_run(A, dA, 4, layout, nv, 0.0, cfg=D.Config(alg=4, chunk=chunk)))


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_not_finite(mats, bad):
    for name in ("short", "hub"):
        A, dA = mats[name]
        for layout in (0, 1):
            for nv in (1, 3, 4, 8):
                B, _, C = _run(A, dA, 4, layout, nv, 0.0, bad=bad)
                want = O.spmm_f32(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
                np.testing.assert_array_equal(np.isfinite(C), np.isfinite(want))
                odd = ~np.isfinite(want)
                np.testing.assert_array_equal(C[odd], want[odd])


# (rows, average row length, columns): on both sides of each line of the rule that
# gives a reference algorithm to the balanced product, by algorithm and layout
_RULE = [(3000, 6, 1), (3000, 6, 16), (3000, 6, 128), (3000, 2, 16), (3000, 2, 64),
         (70000, 2, 16), (70000, 2, 64), (70000, 6, 1), (70000, 6, 64), (70000, 2, 128)]


def _pays(alg, cm, nr, nnz, nv):
    out, sparse = nr * nv, nnz < 4 * nr
    if alg == 0:
        return nv >= 16 and out >= 2**22 if cm else nv >= 32 and out >= 2**23
    if alg == 1:
        return nr >= 65536 or out >= (2**18 if cm else 2**21)
    if alg == 2:
        return cm or nv <= 8 or nv >= 64 or not sparse or out >= 2**23
    if nv <= 8:
        return cm and nv > 1 or nnz < 2**22
    return cm or out >= (2**23 if sparse else 2**18) or (not sparse and nv >= 64)


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nr,deg,nv", _RULE)
def test_reference_algorithms(cuda, nr, deg, nv, layout):
    A = D.gen_random(nr, nr, float(deg), seed=nr + deg)
    dA = D.DeviceCsr(A)
    for beta in (0.0, 0.5):
        want = _run(A, dA, 4, layout, nv, beta)[2]
        for alg in range(4):
            B, C0, C = _run(A, dA, alg, layout, nv, beta)
            _check(A, layout, nv, beta, B, C0, C)
            if _pays(alg, layout == 1, A.nr, A.nnz, nv):
                np.testing.assert_array_equal(C, want)


def test_coo_scalar_keeps_its_chunk(cuda):
    for nv, chunk in ((4, 32), (16, 32), (31, 128), (64, 64), (128, 128)):
        assert D.default_config(2, 0, 1000, 1000, 8000, nv).chunk == chunk


def test_inside_a_capture_they_keep_their_own_kernels(mats):
    """A captured CSR call uses no workspace, so the graph stays good whatever later
    calls do with the library's."""
    import torch
    A, dA = mats["short"]
    st = torch.cuda.Stream()
    for layout in (0, 1):
        nv = 16
        B = torch.rand(A.nc * nv, device="cuda")
        C = torch.empty(A.nr * nv, device="cuda")
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            D.spmm(D.Alg.CSR_SCALAR, layout, dA, B, C, nv=nv, stream=st)
        big = D.DeviceCsr(D.gen_uniform(20000, 20000, 8, seed=1))
        Bb, Cb = (torch.zeros(20000 * 128, device="cuda") for _ in range(2))
        D.spmm(D.Alg.CSR_BALANCED, layout, big, Bb, Cb, nv=128, stream=st)
        C.fill_(float("nan"))
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        c64, absc = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B.cpu().numpy(), nv)
        assert O.rel_err(C.cpu().numpy(), c64, absc) <= O.REL_TOL_F32


def test_no_room_for_copies(cuda):
    """Column-major operands whose copies would take more than the library keeps."""
    import torch
    n, nv = 3_000_000, 96
    rows = np.arange(0, n, 3000)
    lens = np.zeros(n, np.int64)
    lens[rows] = 1
    A = D.Csr(n, n, np.concatenate([[0], np.cumsum(lens)]).astype(np.int32),
              rows.astype(np.int32), np.full(rows.size, 2.0, np.float32))
    dA = D.DeviceCsr(A)
    B = torch.rand(nv, n, device="cuda")
    C = torch.full((nv, n), 3.0, device="cuda")
    D.spmm(D.Alg.CSR_VECTOR, 1, dA, B, C, nv=nv)
    want = torch.zeros(nv, n, device="cuda")
    at = torch.from_numpy(rows).cuda()
    want[:, at] = 2.0 * B[:, at]
    assert torch.equal(C, want)
