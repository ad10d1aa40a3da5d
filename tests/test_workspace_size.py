"""A caller's workspace of exactly daspmm_workspace_bytes suffices wherever B and C lie.

The size is asked for without addresses, so with the widest vectors; operands off
their alignment run with narrower ones.  The host test runs the argument path alone
(no device: a call that is given enough room ends in a CUDA error)."""
import ctypes

import numpy as np
import pytest

import daspmm as D

ERR_CUDA, ERR_WORKSPACE = 3, 5
SIZES = [(4096, 8192), (120_000, 360_000), (262_144, 786_432), (262_144, 1_240_000),
         (1_048_576, 2_000_000)]


def _status(cfg, nr, nnz, nv, ws_bytes, off_b, off_c):
    p = [ctypes.c_void_p(x << 20) for x in range(1, 8)]
    return D.lib().daspmm_spmm_ex(
        ctypes.byref(cfg), 0, nr, nr, nnz, nv, p[0], None, p[1], p[2],
        ctypes.c_void_p(p[3].value + off_b), ctypes.c_void_p(p[4].value + off_c),
        ctypes.c_float(0.0), p[5], ws_bytes, None)


def test_sized_without_addresses():
    import torch
    if torch.cuda.is_available():
        pytest.skip("made-up addresses")
    cfg = D.Config(alg=4)
    bad = []
    for nr, nnz in SIZES:
        for nv in [*range(9, 130), 132, 160, 192, 224, 256, 320, 512]:
            ws = D.workspace_bytes(cfg, 0, nr, nr, nnz, nv)
            for off in ((0, 0), (4, 0), (8, 0), (16, 0), (0, 4), (0, 8), (4, 8)):
                if _status(cfg, nr, nnz, nv, ws, *off) != ERR_CUDA:
                    bad.append((nr, nnz, nv, off))
    assert not bad, f"{len(bad)} refused, first {bad[:5]}"
    assert _status(cfg, 120_000, 360_000, 40, 4096, 0, 0) == ERR_WORKSPACE


@pytest.mark.gpu
@pytest.mark.parametrize("nv", [32, 36, 40, 48, 96])
@pytest.mark.parametrize("off", [1, 2])
def test_runs_in_it(cuda, nv, off):
    import torch
    from oracle import oracle as O
    A = D.gen_random(120_000, 120_000, 3.0, seed=nv)
    dA = D.DeviceCsr(A)
    cfg = D.Config(alg=4)
    ws = torch.zeros(D.workspace_bytes(cfg, 0, A.nr, A.nc, A.nnz, nv), dtype=torch.uint8,
                     device="cuda")
    B = D.gen_dense(A.nc * nv, seed=nv)
    Bt = torch.zeros(B.size + 4, device="cuda")[off:off + B.size]
    Bt.copy_(torch.from_numpy(B))
    C = torch.full((A.nr * nv,), float("nan"), device="cuda")
    D.spmm(4, 0, dA, Bt, C, nv=nv, cfg=cfg, workspace=ws)
    c64, absc = O.spmm_f64(0, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    assert O.rel_err(C.cpu().numpy(), c64, absc) <= O.REL_TOL_F32
