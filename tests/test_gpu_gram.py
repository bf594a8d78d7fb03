"""
The Gram behind tvbg_fc and tvbg_fcfit_loss (csrc/tvbg_gram.cuh: exact
products of fixed-point digits) against a two-pass Pearson in extended
precision, at the edges of its tiles, chunks and paths.

Tolerances: a correlation is rounded once to float32 (2^-24 at |r| <= 1, 1e-7
here); the error sum keeps FP64 and takes about 2^-50 per correlation, 1e-12
of the sum.
"""

import numpy as np
import pytest

from tvb_hpc import metric

pytestmark = pytest.mark.gpu


def pearson(x):
    x = x.astype(np.longdouble)
    c = x - x.mean(axis=1, keepdims=True)
    g = np.einsum('bti,btj->bij', c, c)
    s = np.sqrt(np.einsum('bii->bi', g))
    with np.errstate(all='ignore'):
        return g / (s[:, :, None] * s[:, None, :])


def series(I, T, N, seed, mean=1.0, std=0.05):
    rng = np.random.default_rng(seed)
    x = np.cumsum(rng.normal(size=(I, T, 3)), 1) @ rng.normal(size=(I, 3, N)) + rng.normal(size=(I, T, N))
    return (mean + std * x).astype(np.float32)


def check(cuda, x):
    torch = cuda
    I, T, N = x.shape
    tg = np.corrcoef(np.random.default_rng(N).normal(size=(max(2, N), 50))).astype(np.float32)[:N, :N].copy()
    fc, err = metric.fc(torch.from_numpy(x).cuda(), torch.from_numpy(tg).cuda())
    ref = pearson(x)
    fc, err = fc.cpu().numpy(), err.cpu().numpy()
    np.testing.assert_array_equal(np.isnan(fc), np.isnan(ref.astype(np.float32)))
    ok = ~np.isnan(ref)
    assert np.abs(fc[ok] - ref[ok]).max(initial=0) < 1e-7
    assert np.array_equal(fc, fc.transpose(0, 2, 1), equal_nan=True)
    iu = np.triu_indices(N, 1)
    e = ((ref - tg)[:, iu[0], iu[1]] ** 2).sum(-1)
    np.testing.assert_allclose(err, e.astype(np.float64), rtol=1e-12, equal_nan=True)


@pytest.mark.parametrize('I,T,N', [(1, 2, 1), (3, 2, 2), (2, 15, 15), (2, 16, 16), (2, 17, 17),
                                   (1, 63, 95), (2, 64, 96), (1, 65, 97), (2, 130, 127),
                                   (1, 129, 128), (2, 65, 129), (1, 200, 193), (1, 40, 400),
                                   (1, 20, 2050), (200, 40, 84)])
def test_fc_edges(cuda, I, T, N):
    check(cuda, series(I, T, N, seed=T + N))


@pytest.mark.parametrize('N', [20, 140])
@pytest.mark.parametrize('mean,std', [(1e4, 0.5), (-3.0, 1e-5), (0.0, 1e-30), (0.0, 1e-38),
                                      (0.0, 1e35), (2e37, 1e36)])
def test_fc_scales(cuda, N, mean, std):
    check(cuda, series(2, 150, N, seed=9, mean=mean, std=std))


@pytest.mark.parametrize('N', [20, 140])
def test_fc_constant_and_nonfinite_nodes(cuda, N):
    x = series(2, 70, N, seed=4)
    x[0, :, 3] = 0.25            # constant: no correlation
    x[0, 7, 5] = np.nan
    x[1, 9, 0] = np.inf
    x[1, :, N - 1] = 0.0
    check(cuda, x)
