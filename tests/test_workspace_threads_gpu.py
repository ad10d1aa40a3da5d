"""The library's workspaces under several threads: a block that another thread's call
makes larger is not taken from under one that uses it, and a stream whose block grows
does not hold up the others."""
import threading
import time

import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_one_stream_many_threads(cuda):
    import torch
    A = D.gen_powerlaw(20000, seed=3)
    dA = D.DeviceCsr(A)
    st = torch.cuda.Stream()
    want_own = D.ownership(4, dA, 64, 32).cpu().numpy()
    want_fp = D.fingerprint(0, dA, 64)
    seen, errors = [], []

    def look():
        try:
            for _ in range(40):
                own = D.ownership(4, dA, 64, 32, stream=st)
                seen.append((own, D.fingerprint(0, dA, 64, stream=st)))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    def grow():
        try:
            for nv in (32, 64, 96, 128, 160, 256, 512):   # each needs a larger block
                B = torch.zeros(A.nc * nv, device="cuda")
                C = torch.empty(A.nr * nv, device="cuda")
                torch.cuda.current_stream().synchronize()
                D.spmm(4, 0, dA, B, C, nv=nv, stream=st)
                st.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=f) for f in (look, grow)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    torch.cuda.synchronize()
    for own, fp in seen:
        np.testing.assert_array_equal(own.cpu().numpy(), want_own)
        assert fp == want_fp


def test_growth_holds_up_its_own_stream_only(cuda):
    import torch
    A = D.gen_uniform(4096, 4096, 8, seed=1)
    dA = D.DeviceCsr(A)
    busy, free = torch.cuda.Stream(), torch.cuda.Stream()
    nv, big = 32, 512
    B, C = (torch.rand(4096 * nv, device="cuda") for _ in range(2))
    Bb, Cb = (torch.rand(4096 * big, device="cuda") for _ in range(2))
    large = D.DeviceCsr(D.gen_uniform(4096, 4096, 256, seed=2))
    for st in (busy, free):
        D.spmm(4, 0, dA, B, C, nv=nv, stream=st)
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(4_000_000_000)   # about two seconds
    t = threading.Thread(target=lambda: D.spmm(4, 0, large, Bb, Cb, nv=big, stream=busy))
    t.start()
    time.sleep(0.3)            # it waits for the busy stream before it frees its block
    assert t.is_alive()
    t0 = time.perf_counter()
    D.spmm(4, 0, dA, B, C, nv=nv, stream=free)
    free.synchronize()
    assert time.perf_counter() - t0 < 0.5
    t.join()
    torch.cuda.synchronize()
    c64, absc = O.spmm_f64(0, 4096, 4096, A.rowPtr, A.colIdx, A.values, B.cpu().numpy(), nv)
    assert O.rel_err(C.cpu().numpy(), c64, absc) <= O.REL_TOL_F32
