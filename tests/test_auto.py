"""DASPMM_ALG_AUTO where nothing has been tuned: below 32 columns and for column-major
operands it needs no workspace, and so runs where none can be had (inside a capture,
operands whose copies would not fit), in its own kernel there."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O


@pytest.mark.parametrize("layout,nv", [(0, 1), (0, 8), (0, 16), (0, 31), (1, 1), (1, 16), (1, 128)])
def test_its_configuration_needs_no_workspace(layout, nv):
    D.lib().daspmm_tune_clear()
    for nr, nnz in ((1000, 8000), (262_144, 1_240_000), (262_144, 1000)):
        cfg = D.default_config(D.Alg.AUTO, layout, nr, nr, nnz, nv)
        assert D.workspace_bytes(cfg, layout, nr, nr, nnz, nv) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("layout,nv", [(0, 1), (0, 16), (1, 1), (1, 32)])
def test_inside_a_capture(cuda, layout, nv):
    import torch
    D.lib().daspmm_tune_clear()
    A = D.gen_powerlaw(100_000, mean_scale=1.7, seed=5)
    dA = D.DeviceCsr(A)
    B = D.gen_dense(A.nc * nv, seed=nv)
    Bt, C = torch.from_numpy(B).cuda(), torch.zeros(A.nr * nv, device="cuda")
    c64, absc = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)

    def right():
        torch.cuda.synchronize()
        assert O.rel_err(C.cpu().numpy(), c64, absc) <= O.REL_TOL_F32
        C.fill_(float("nan"))
        torch.cuda.synchronize()

    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for first in (True, False):   # a stream that the library has not seen, and one it has
        g = torch.cuda.CUDAGraph()
        n = D.lib().daspmm_launch_count()
        with torch.cuda.graph(g, stream=st):
            D.spmm(D.Alg.AUTO, layout, dA, Bt, C, nv=nv, stream=st)
        assert D.lib().daspmm_launch_count() - n == 1   # CSR scalar
        D.spmm(D.Alg.AUTO, layout, dA, Bt, C, nv=nv, stream=st)
        right()
        big = D.DeviceCsr(D.gen_uniform(120_000, 120_000, 16, seed=1))
        Bb, Cb = (torch.zeros(120_000 * 64, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        for alg in (D.Alg.AUTO, D.Alg.CSR_BALANCED):
            D.spmm(alg, 1, big, Bb, Cb, nv=64, stream=st)
        torch.cuda.synchronize()
        D.lib().daspmm_scratch_trim(0)
        g.replay()
        right()


@pytest.mark.gpu
def test_no_room_for_copies(cuda):
    import torch
    D.lib().daspmm_tune_clear()
    n, nv = 3_000_000, 96
    rows = np.arange(0, n, 3000)
    lens = np.zeros(n, np.int64)
    lens[rows] = 1
    A = D.Csr(n, n, np.concatenate([[0], np.cumsum(lens)]).astype(np.int32),
              rows.astype(np.int32), np.full(rows.size, 2.0, np.float32))
    B = torch.rand(nv, n, device="cuda")
    C = torch.full((nv, n), 3.0, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    D.spmm(D.Alg.AUTO, 1, D.DeviceCsr(A), B, C, nv=nv)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 256 << 20
    want = torch.zeros(nv, n, device="cuda")
    at = torch.from_numpy(rows).cuda()
    want[:, at] = 2.0 * B[:, at]
    assert torch.equal(C, want)
