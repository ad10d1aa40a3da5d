"""The vector and the one-by-one forms of the device quantizers: element counts
around the vector width, addresses off its alignment, column counts that a
vector of eight divides or not, NaN and infinities -- bit for bit against the
oracle's conversions and the column maxima of numpy."""
import numpy as np
import pytest

import daspmm as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _codes(q):
    import torch
    return (q if q.dtype == torch.uint8 else q.view(torch.int16)).cpu().numpy()


def _want(fmt, x):
    w = O.quantize(int(fmt), x)
    return w if fmt == D.Fmt.E4M3 else w.view(np.int16)


@pytest.mark.parametrize("fmt", [D.Fmt.BF16, D.Fmt.F16, D.Fmt.E4M3])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 24, 2048 * 8 + 8, 700001, 8 * 1_300_000])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_plain(cuda, fmt, n, off):
    import torch
    x = np.random.default_rng(n).normal(0, 3, n + off).astype(np.float32)
    xt = torch.from_numpy(x).cuda()[off:]
    np.testing.assert_array_equal(_codes(D.quantize(xt, fmt)), _want(fmt, x[off:]))


@pytest.mark.parametrize("rows,cols", [(1, 8), (3, 5), (500, 12), (9001, 24), (2, 70000),
                                       (65536, 40), (4097, 256), (33, 1)])
@pytest.mark.parametrize("off", [0, 1])
def test_scaled(cuda, rows, cols, off):
    import torch
    rng = np.random.default_rng(rows)
    B = (rng.normal(0, 1, (rows, cols)) * rng.uniform(0.01, 50, cols)).astype(np.float32)
    B[:, 0] = 0.0
    flat = np.concatenate([np.zeros(off, np.float32), B.reshape(-1)])
    Bt = torch.from_numpy(flat).cuda()[off:]
    sc = D.e4m3_scales(Bt, rows, cols)
    top = np.abs(B).max(axis=0)
    want = np.where(top > 0, top / np.float32(448.0), np.float32(1.0)).astype(np.float32)
    np.testing.assert_array_equal(sc.cpu().numpy(), want)
    q = D.quantize(Bt, D.Fmt.E4M3, sc, cols)
    np.testing.assert_array_equal(_codes(q).reshape(rows, cols),
                                  O.quantize(3, (B / want).astype(np.float32)).reshape(rows, cols))


def test_not_finite(cuda):
    import torch
    x = np.array([np.inf, -np.inf, np.nan, 1e30, -1e30, 0.0, -0.0, 1.0] * 3, np.float32)
    a, b = torch.from_numpy(x).cuda(), torch.from_numpy(np.append(x, 0.0)).cuda().float()
    for fmt in (D.Fmt.BF16, D.Fmt.F16, D.Fmt.E4M3):
        # 24 elements take the vector form, 25 the one-by-one form
        np.testing.assert_array_equal(_codes(D.quantize(a, fmt)), _codes(D.quantize(b, fmt))[:24])
