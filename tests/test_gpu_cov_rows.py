"""
Streaming FC in several rows per call (tvbg_cov_update_rows) against numpy in
FP64, at the edges of its tiles (32 nodes), passes (16 samples, fewer for
large N) and CTA parts; chunked calls, strided, negative and repeated rows.

Tolerance: FP64 sums of at most 40 products, 40 * 2^-52 < 1e-13 of the sum of
magnitudes; the correlation is rounded to float32 (1e-7).
"""

import numpy as np
import pytest

from tvb_hpc import metric

pytestmark = pytest.mark.gpu


def check(fc, x):
    x = x.astype(np.float64)
    u = x - x.mean(axis=1, keepdims=True)
    ref = np.einsum('bti,btj->bij', u, u)
    mag = np.sqrt(np.einsum('bii->bi', ref))
    mag = mag[:, :, None] * mag[:, None, :]
    m2 = fc.m2.cpu().numpy()
    assert np.all(np.abs(m2 - ref) <= 1e-13 * mag * x.shape[1])
    assert np.array_equal(m2, m2.transpose(0, 2, 1))
    np.testing.assert_allclose(fc.corr().cpu().numpy(), ref / mag, atol=1e-7)


@pytest.mark.parametrize('I,N', [(1, 1), (3, 31), (2, 32), (2, 33), (700, 5), (40, 84), (2, 300),
                                 (1, 1025)])
@pytest.mark.parametrize('split', [(40, ), (1, 15, 16, 8), (17, 1, 22)])
def test_rows(cuda, I, N, split):
    torch = cuda
    x = (1.0 + 0.1 * np.random.default_rng(N).normal(size=(I, 40, N))).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    fc = metric.StreamingFC(I, N)
    r = 0
    for n in split:
        fc.update_rows(xd, range(r, r + n))
        r += n
    assert fc.n == 40
    check(fc, x)
    np.testing.assert_allclose(fc.mean.cpu().numpy(), x.astype(np.float64).mean(axis=1), rtol=1e-14)


@pytest.mark.parametrize('rows', [range(0, 40, 3), range(39, -1, -1), [-1, -3, -5], [4, 4, 4, 7],
                                  [0, 1, 5, 2]])
def test_row_orders(cuda, rows):
    torch = cuda
    x = np.random.default_rng(1).normal(size=(4, 40, 50)).astype(np.float32)
    fc = metric.StreamingFC(4, 50)
    fc.update_rows(torch.from_numpy(x).cuda(), rows)
    check(fc, x[:, list(rows), :])
    wide = torch.from_numpy(np.concatenate([x, x], 2)).cuda()[:, :, :50]   # strided samples
    fc = metric.StreamingFC(4, 50)
    fc.update_rows(wide, rows)
    check(fc, x[:, list(rows), :])


def test_row_out_of_range(cuda):
    fc = metric.StreamingFC(2, 5)
    with pytest.raises(IndexError):
        fc.update_rows(cuda.zeros((2, 3, 5), device='cuda'), [1, 3])
