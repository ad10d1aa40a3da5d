"""Calls of the reference's algorithms that run as the balanced product: what they do to
memory, captures, streams and threads of the caller."""
import threading

import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# (algorithm, layout, N) of calls that the balanced product takes at 20,000 rows of 8
ROUTED = [(D.Alg.CSR_VECTOR, 1, 32), (D.Alg.COO_SCALAR, 0, 64), (D.Alg.CSR_VECTOR, 0, 128)]


@pytest.fixture(scope="module")
def mat(cuda):
    A = D.gen_powerlaw(20000, mean_scale=1.7, seed=5)
    return A, D.DeviceCsr(A)


def _beta(alg):
    return 1.0 if alg in (D.Alg.COO_SCALAR, D.Alg.COO_VECTOR) else 0.0


def _launches(f):
    import torch
    torch.cuda.synchronize()
    n = D.lib().daspmm_launch_count()
    f()
    torch.cuda.synchronize()
    return D.lib().daspmm_launch_count() - n


def _operands(A, nv):
    import torch
    B = D.gen_dense(A.nc * nv, seed=nv)
    Bt, C = torch.from_numpy(B).cuda(), torch.zeros(A.nr * nv, device="cuda")
    torch.cuda.synchronize()   # the calls are on other streams
    return B, Bt, C


def _check(A, layout, nv, B, C):
    c64, absc = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values, B, nv)
    assert O.rel_err(C.cpu().numpy(), c64, absc) <= O.REL_TOL_F32


@pytest.mark.parametrize("alg,layout,nv", ROUTED)
def test_own_kernels_inside_a_capture(mat, alg, layout, nv):
    """Outside a capture such a call launches the balanced product's kernels, inside one
    its own; the graph stays good when later calls need more memory."""
    import torch
    A, dA = mat
    st = torch.cuda.Stream()
    B, Bt, C = _operands(A, nv)
    D.spmm(alg, layout, dA, Bt, C, beta=_beta(alg), nv=nv, stream=st,   # (COO: the workspace)
           cfg=D.Config(alg=int(alg)))
    own = _launches(lambda: D.spmm(alg, layout, dA, Bt, C, beta=_beta(alg), nv=nv, stream=st,
                                   cfg=D.Config(alg=int(alg))))
    routed = _launches(lambda: D.spmm(alg, layout, dA, Bt, C, beta=_beta(alg), nv=nv, stream=st))
    assert routed != own
    g = torch.cuda.CUDAGraph()
    n = D.lib().daspmm_launch_count()
    with torch.cuda.graph(g, stream=st):
        D.spmm(alg, layout, dA, Bt, C, beta=_beta(alg), nv=nv, stream=st)
    assert D.lib().daspmm_launch_count() - n == own
    big = D.DeviceCsr(D.gen_uniform(60000, 60000, 8, seed=1))
    Bb, Cb = (torch.zeros(60000 * 128, device="cuda") for _ in range(2))
    D.spmm(D.Alg.CSR_VECTOR, 1, big, Bb, Cb, nv=128, stream=st)
    torch.cuda.synchronize()
    D.lib().daspmm_scratch_trim(0)
    C.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    _check(A, layout, nv, B, C)


@pytest.mark.parametrize("alg,layout,nv", ROUTED)
def test_while_another_stream_is_captured(mat, alg, layout, nv):
    """A call on another stream than the one that this thread captures allocates without
    ending the capture, the first time too."""
    import torch
    A, dA = mat
    st, other = torch.cuda.Stream(), torch.cuda.Stream()
    B, Bt, C = _operands(A, nv)
    B2, Bt2, C2 = _operands(A, nv)
    D.spmm(alg, layout, dA, Bt, C, nv=nv, stream=other,   # COO: the workspace is there
           cfg=D.Config(alg=int(alg)))
    D.spmm(D.Alg.CSR_SCALAR, layout, dA, Bt, C, nv=nv, stream=st, cfg=D.Config(alg=0))
    torch.cuda.synchronize()
    C.zero_()
    torch.cuda.synchronize()
    D.lib().daspmm_scratch_trim(0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        D.spmm(D.Alg.CSR_SCALAR, layout, dA, Bt2, C2, nv=nv, stream=st, cfg=D.Config(alg=0))
        D.spmm(alg, layout, dA, Bt, C, beta=_beta(alg), nv=nv, stream=other)
    g.replay()
    torch.cuda.synchronize()
    _check(A, layout, nv, B, C)
    _check(A, layout, nv, B2, C2)


@pytest.mark.parametrize("alg", [D.Alg.COO_SCALAR, D.Alg.COO_VECTOR])
@pytest.mark.parametrize("layout,nv", [(0, 4), (0, 64), (1, 32)])
def test_captured_after_the_same_call(mat, alg, layout, nv):
    """The call before a capture leaves what the captured one needs (COO's own kernels
    have a workspace), though it ran as the balanced product itself."""
    import torch
    A, dA = mat
    st = torch.cuda.Stream()
    B, Bt, C = _operands(A, nv)
    D.spmm(alg, layout, dA, Bt, C, beta=1.0, nv=nv, stream=st)
    torch.cuda.synchronize()
    _check(A, layout, nv, B, C)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        D.spmm(alg, layout, dA, Bt, C, beta=1.0, nv=nv, stream=st)
    C.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    _check(A, layout, nv, B, C)


def test_memory_is_given_back(mat):
    import torch
    A, dA = mat
    nv = 256
    _, Bt, C = _operands(A, nv)
    D.spmm(D.Alg.CSR_VECTOR, 1, dA, Bt, C, nv=nv)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    assert D.lib().daspmm_scratch_trim(0) == 0
    assert torch.cuda.mem_get_info()[0] >= held + 8 * A.nr * nv * 3 // 4
    D.spmm(D.Alg.CSR_VECTOR, 1, dA, Bt, C, nv=nv)
    torch.cuda.synchronize()


def test_threads_on_streams_of_their_own_and_one_stream(mat):
    import torch
    A, dA = mat
    shared = torch.cuda.Stream()
    out, errors = [], []

    def work(i):
        try:
            st = shared if i % 2 else torch.cuda.Stream()
            for k in range(12):
                alg, layout, nv = ROUTED[(i + k) % len(ROUTED)]
                with torch.cuda.stream(st):
                    Bt = torch.from_numpy(D.gen_dense(A.nc * nv, seed=nv)).cuda()
                    C = torch.zeros(A.nr * nv, device="cuda")
                    st.synchronize()
                D.spmm(alg, layout, dA, Bt, C, beta=_beta(alg), nv=nv, stream=st)
                out.append((layout, nv, Bt, C))
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    want = {}
    for layout, nv, Bt, C in out:
        key = (layout, nv)
        if key not in want:
            want[key] = O.spmm_f64(layout, A.nr, A.nc, A.rowPtr, A.colIdx, A.values,
                                   Bt.cpu().numpy(), nv)
        assert O.rel_err(C.cpu().numpy(), *want[key]) <= O.REL_TOL_F32
    np.testing.assert_equal(len(out), 48)


def test_a_large_call_repeated_after_a_synchronisation(cuda):
    """What the pool keeps covers the largest call that it serves: the second call finds
    its memory mapped (mapping 1.2 GB takes milliseconds, the call about 0.5)."""
    import time
    import torch
    n, nv = 1 << 20, 144
    A = D.gen_uniform(n, n, 1, seed=1)
    dA = D.DeviceCsr(A)
    B, C = (torch.zeros(n * nv, device="cuda") for _ in range(2))
    took = []
    for _ in range(8):
        torch.cuda.synchronize()
        t = time.perf_counter()
        D.spmm(D.Alg.CSR_VECTOR, 1, dA, B, C, nv=nv)
        torch.cuda.synchronize()
        took.append(time.perf_counter() - t)
    D.lib().daspmm_scratch_trim(0)
    assert sorted(took[1:])[3] < 3e-3, took
