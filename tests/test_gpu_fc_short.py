"""
Pearson FC of few nodes and short series (FP64 sums), on both sides of the line
to the digit products, against extended precision.

Tolerances: a correlation takes one float32 rounding (1e-7), the error sum 1e-12
of itself.
"""

import numpy as np
import pytest

from tvb_hpc import metric

pytestmark = pytest.mark.gpu


# N: samples on the line (T (N^2 + 300) <= 70000) and one more; 51 nodes never take FP64 sums
@pytest.mark.parametrize('N,T', [(N, T) for N in (1, 2, 10, 31, 32, 45, 50) for T in
                                 sorted({2, 31, 33, 70000 // (N * N + 300), 70000 // (N * N + 300) + 1})]
                         + [(51, 2), (51, 17)])
def test_short_series(cuda, N, T):
    torch = cuda
    rng = np.random.default_rng(N + T)
    I = 3
    x = rng.normal(1.0, 0.3, (I, T, N)).astype(np.float32)
    target = rng.uniform(-1, 1, (N, N)).astype(np.float32)
    fc, err = metric.fc(torch.from_numpy(x).cuda(), torch.from_numpy(target).cuda())
    u = x.astype(np.longdouble)
    u = u - u.mean(axis=1, keepdims=True)
    g = np.einsum('bti,btj->bij', u, u)
    s = np.sqrt(np.einsum('bii->bi', g))
    ref = g / (s[:, :, None] * s[:, None, :])
    got = fc.cpu().numpy()
    assert np.abs(got - ref).max() <= 1e-7
    np.testing.assert_array_equal(got, got.transpose(0, 2, 1))
    iu = np.triu_indices(N, 1)
    e = ((ref - target)[:, iu[0], iu[1]]**2).sum(axis=1)
    assert np.all(np.abs(err.cpu().numpy() - e) <= 1e-12 * np.maximum(e, 1e-300) + 1e-14)
    # a constant and an infinite node have no correlations, the others keep theirs
    if N >= 4:
        x[:, :, 1] = np.float32(0.3)
        x[0, 0, 2] = np.inf
        got = metric.fc(torch.from_numpy(x).cuda(), torch.from_numpy(target).cuda())[0].cpu().numpy()
        bad = np.zeros((I, N), bool)
        bad[:, 1] = True
        bad[0, 2] = True
        np.testing.assert_array_equal(np.isnan(got), bad[:, :, None] | bad[:, None, :])
        keep = ~(bad[:, :, None] | bad[:, None, :])
        assert np.abs(got[keep] - ref[keep]).max() <= 1e-7
