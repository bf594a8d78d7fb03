"""
Constant nodes in long series: the mean is the constant itself at any length,
so such a node has no correlation (NaN) on every path of tvbg_gram.cuh, and a
node of the other kind keeps its correlations.  Constants without a short
binary fraction, lengths at the edges of the runs of samples that a mean sums
in FP32 words (256 per thread, two threads a node) and far beyond.

Tolerance: correlations are rounded to float32 (1e-7); FP64 reference.
"""

import ctypes

import numpy as np
import pytest

from tvb_hpc import metric, _native as nat

pytestmark = pytest.mark.gpu


def series(T, N, seed):
    "The first third of the nodes constant, the rest noise; and the mask of the constant ones."
    rng = np.random.default_rng(seed)
    x = rng.normal(1.0, 0.3, size=(T, N)).astype(np.float32)
    nc = N // 3
    x[:, :nc] = rng.uniform(0.01, 1.99, nc).astype(np.float32)
    x[:, nc - 1] = np.float32(-3.1e-5)
    return x, np.arange(N) < nc


def check(fc, x, const):
    bad = const[:, None] | const[None, :]
    np.testing.assert_array_equal(np.isnan(fc), bad)
    ref = np.corrcoef(x[:, ~const].astype(np.float64).T)
    assert np.abs(fc[np.ix_(~const, ~const)] - ref).max() < 1e-7


@pytest.mark.parametrize('T', [511, 512, 513, 1025, 20000, 200000])
@pytest.mark.parametrize('N', [20, 100, 140])
def test_constant_nodes(cuda, T, N):
    torch = cuda
    x, const = series(T, N, T + N)
    target = torch.zeros(N, N, device='cuda')
    fc, err = metric.fc(torch.from_numpy(x[None]).cuda(), target)
    check(fc[0].cpu().numpy(), x, const)
    assert bool(torch.isnan(err).all())


@pytest.mark.parametrize('T', [513, 20000, 60000])
def test_constant_nodes_in_the_loss_path(cuda, T):
    torch = cuda
    lib = nat.load()
    N = 200          # above 192 nodes: digit products
    x, const = series(T, N, T)
    xd = torch.from_numpy(x).cuda()
    target = torch.eye(N, dtype=torch.float64, device='cuda')
    nb = ctypes.c_int64()
    nat.check(lib.tvbg_fcfit_scratch_bytes(1, N, ctypes.byref(nb)))
    scratch = torch.empty(nb.value, dtype=torch.uint8, device='cuda')
    loss = torch.empty(1, dtype=torch.float64, device='cuda')
    fc = torch.empty(N, N, dtype=torch.float64, device='cuda')
    nat.check(lib.tvbg_fcfit_loss(xd.data_ptr(), T * N, None, 0, 0, 1, 1, T, N, target.data_ptr(),
                                  loss.data_ptr(), None, 0, fc.data_ptr(), scratch.data_ptr(), None))
    torch.cuda.synchronize()
    check(fc.cpu().numpy(), x, const)
    assert bool(torch.isnan(loss).all())
