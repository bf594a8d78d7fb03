"""
Co-moment updates by one sample, and correlations of few nodes in many
instances; on both sides of the lines of their dispatch.

Tolerances: an update by one sample takes the same operations as one by several (equal
bits), FP64 against numpy 1e-13 of the sum of magnitudes and sample; a
correlation takes one float32 rounding (1e-7).
"""

import ctypes

import numpy as np
import pytest

from tvb_hpc import metric, _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,N', [(1, 1), (3, 7), (5, 33), (2, 100), (2, 101), (700, 101), (599, 32), (600, 32), (600, 33), (9, 140), (2, 3000)])
def test_one_sample_updates(cuda, I, N):
    torch = cuda
    rng = np.random.default_rng(N)
    x = (1.0 + 0.1 * rng.normal(size=(I, 6, N))).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    one, two = metric.StreamingFC(I, N), metric.StreamingFC(I, N)
    for k in range(6):
        one.update(xd[:, k])
    two.update_rows(xd, [0, 1])
    two.update_rows(xd, [2])
    two.update_rows(xd, [3, 4, 5])
    assert torch.equal(one.mean, two.mean)
    assert torch.equal(one.m2, two.m2)
    assert torch.equal(one.m2, one.m2.transpose(1, 2))
    u = x.astype(np.float64)
    u -= u.mean(axis=1, keepdims=True)
    s = np.sqrt(np.einsum('bti,bti->bi', u, u))
    for b in (0, I - 1):
        assert np.all(np.abs(one.m2[b].cpu().numpy() - u[b].T @ u[b]) <= 6e-13 * s[b][:, None] * s[b][None, :])


@pytest.mark.parametrize('I', [1, 9, 399, 400, 999, 1000])
@pytest.mark.parametrize('N', [1, 2, 6, 7, 16, 17, 24, 25, 32, 33])
def test_small_correlations(cuda, I, N):
    torch = cuda
    rng = np.random.default_rng(N * I)
    a = rng.normal(size=(I, N, N + 3))
    m2 = a @ a.transpose(0, 2, 1)
    m2[:, 0] = m2[:, :, 0] = 0.0        # a constant node: no correlation
    corr = torch.full((I, N, N), 7.0, device='cuda')
    m2d = torch.from_numpy(m2).cuda()
    nat.check(nat.load().tvbg_cov_corr(m2d.data_ptr(), I, N, corr.data_ptr(),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = corr.cpu().numpy()
    assert np.isnan(got[:, 0]).all() and np.isnan(got[:, :, 0]).all()
    s = np.sqrt(np.einsum('bii->bi', m2))[:, 1:]
    assert np.all(np.abs(got[:, 1:, 1:] - m2[:, 1:, 1:] / (s[:, :, None] * s[:, None, :])) <= 1e-7)
    np.testing.assert_array_equal(got, got.transpose(0, 2, 1))
