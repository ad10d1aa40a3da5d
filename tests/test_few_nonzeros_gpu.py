"""Matrices with far fewer nonzeros than rows: the reference's algorithms and AUTO keep
their own kernels at the widths where the balanced product would seek every row (seen by
the number of launches), and take it for the same rows with more in them."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu
NR = 131_072


def _launches(alg, layout, dA, B, C, nv, cfg=None):
    n = D.lib().daspmm_launch_count()
    D.spmm(alg, layout, dA, B, C, beta=0.0 if alg in (0, 1, 5) else 1.0, nv=nv, cfg=cfg)
    return D.lib().daspmm_launch_count() - n


@pytest.mark.parametrize("layout,nv", [(0, 16), (0, 64), (1, 16), (1, 64)])
def test_who_runs(cuda, layout, nv):
    import torch
    D.lib().daspmm_tune_clear()
    for deg in (0.25, 8.0):
        A = D.gen_random(NR, NR, deg, seed=nv)
        dA = D.DeviceCsr(A)
        B = D.gen_dense(NR * nv, seed=1)
        Bt = torch.from_numpy(B).cuda()
        c64, absc = O.spmm_f64(layout, NR, NR, A.rowPtr, A.colIdx, A.values, B, nv)
        for alg in (0, 1, 2, 3, 5):
            if alg == 5 and layout == 0 and nv >= 32:
                continue   # AUTO's configuration is the balanced product there
            C = torch.zeros(NR * nv, device="cuda")
            n = _launches(alg, layout, dA, Bt, C, nv)
            got = C.cpu().numpy()
            own = _launches(0 if alg == 5 else alg, layout, dA, Bt, C, nv,
                            cfg=D.Config(alg=0 if alg == 5 else alg))
            assert O.rel_err(got, c64, absc) <= O.REL_TOL_F32
            if deg < 1:
                assert n == own, alg
            elif layout == 1 and alg != 0:
                assert n > own, alg


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("nv", [1, 8])
def test_few_columns(cuda, layout, nv):
    import torch
    D.lib().daspmm_tune_clear()
    lens = np.zeros(300_000, int)
    lens[::1049] = 1
    A = D.Csr(lens.size, 5000, np.concatenate([[0], np.cumsum(lens)]).astype(np.int32),
              np.random.default_rng(1).integers(0, 5000, int(lens.sum())).astype(np.int32),
              np.ones(int(lens.sum()), np.float32))
    dA = D.DeviceCsr(A)
    B = D.gen_dense(5000 * nv, seed=1)
    Bt = torch.from_numpy(B).cuda()
    c64, absc = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    for alg in (0, 2, 3, 5):
        C = torch.zeros(A.nr * nv, device="cuda")
        n = _launches(alg, layout, dA, Bt, C, nv)
        got = C.cpu().numpy()
        own = _launches(0 if alg == 5 else alg, layout, dA, Bt, C, nv,
                        cfg=D.Config(alg=0 if alg == 5 else alg))
        assert n == own, alg
        assert O.rel_err(got, c64, absc) <= O.REL_TOL_F32
