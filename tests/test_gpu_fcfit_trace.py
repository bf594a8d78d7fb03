"""
FCFit with the forward's whole trace against checkpoints and recomputation
(the same kernels on the same values: equal bits), on both reverse kernels,
through a change of the memory budget between calls of one problem; and the
loss path on a trace of several values per node against the same series
alone (equal bits).
"""

import ctypes

import numpy as np
import pytest

from tvb_hpc import _native as nat
from tvb_hpc import network, adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,N,T,C', [(1, 20, 41, 20), (8, 40, 250, 30), (19, 84, 203, 100), (9, 130, 64, 100)])
def test_trace_equals_checkpoints(cuda, I, N, T, C):
    torch = cuda
    w, ln = network.synthetic_connectome(N, 0.3, seed=N)
    conn = network.Connectivity.from_dense(w, ln)
    rng = np.random.default_rng(N)
    x0 = np.stack([rng.uniform(0.05, 0.3, (I, N)), rng.uniform(-1.5, -0.5, (I, N))], -1).astype(np.float32)
    eta = rng.uniform(-6, -4, (I, N)).astype(np.float32)
    G = np.linspace(0.3, 0.6, I).astype(np.float32)
    target = np.corrcoef(rng.normal(size=(N, 60))).astype(np.float32)
    prob = adjoint.FCFit(conn, 0.1, 4.0, x0, target, T, checkpoint_every=C)
    assert prob.layout == 'groups' and prob.adjoint_kernel == 'groups' and prob._traced()
    budget = prob.trace_budget
    out = []
    for b, kernel in ((budget, 'groups'), (1, 'groups'), (budget, 'instances'), (1, 'instances'), (budget, 'groups')):
        prob.trace_budget = b
        assert prob._traced() == (b == budget)
        loss = prob.forward(G, eta).clone()
        prob.adjoint_kernel = kernel
        out.append([loss] + [t.clone() for t in prob.backward()])
        prob.adjoint_kernel = 'groups'
    for o in out[1:]:
        assert all(torch.equal(x, y) for x, y in zip(out[0], o))


@pytest.mark.parametrize('N,lanes,cols', [(84, 8, 3), (130, 8, 3), (33, 1, 2)])
def test_loss_columns(cuda, N, lanes, cols):
    torch = cuda
    lib = nat.load()
    rng = np.random.default_rng(3)
    I, T = 11, 70
    g = -(-I // lanes)
    full = torch.from_numpy(rng.standard_normal((g, T, N, cols, lanes)).astype(np.float32)).cuda()
    one = full[:, :, :, 0].contiguous()
    target = torch.from_numpy(np.corrcoef(rng.normal(size=(N, 60)))).cuda()
    nb = ctypes.c_int64()
    nat.check(lib.tvbg_fcfit_scratch_bytes(I, N, ctypes.byref(nb)))
    scratch = torch.empty(int(nb.value), dtype=torch.uint8, device='cuda')
    out = []
    for x, c in ((full, cols), (one, 1)):
        loss = torch.empty(I, dtype=torch.float64, device='cuda')
        dx = torch.empty((I, T, N), device='cuda')
        fc = torch.empty((I, N, N), dtype=torch.float64, device='cuda')
        nat.check(lib.tvbg_fcfit_loss_ex(x.data_ptr(), T * N * c * lanes, c, None, 0, 0, lanes, I, T, N,
                                         target.data_ptr(), loss.data_ptr(), dx.data_ptr(), T * N,
                                         fc.data_ptr(), scratch.data_ptr(), nat.stream_handle()))
        out.append((loss, dx, fc))
    assert all(torch.equal(a, b) for a, b in zip(*out))
    with pytest.raises(nat.TvbgError):
        nat.check(lib.tvbg_fcfit_loss_ex(one.data_ptr(), T * N * lanes, 0, None, 0, 0, lanes, I, T, N,
                                         target.data_ptr(), loss.data_ptr(), dx.data_ptr(), T * N,
                                         fc.data_ptr(), scratch.data_ptr(), nat.stream_handle()))
