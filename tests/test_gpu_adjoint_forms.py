"""
The forms of the lane-interleaved reverse kernel that the model's default
does not reach, against the per-instance kernel on the same traces (equal
bits: the same per-step code and the same out-edge order): tau other than 1;
delays below three blocks, where the CTAs of a cluster wait for each phase
before the next (2 K <= d_min < 3 K); more edges than
the staged records hold; node slots that do not divide among the CTAs.
"""

import numpy as np
import pytest

from tvb_hpc import network, adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N,density,K,tau,near', [
    (41, 0.3, 8, 1.5, False), (41, 0.3, 8, 1.0, True), (84, 0.9, 8, 1.0, False),
    (84, 0.9, 4, 0.7, False), (33, 0.1, 4, 1.0, False)])
@pytest.mark.parametrize('pipe', [True, False])
def test_forms(cuda, N, density, K, tau, near, pipe):
    torch = cuda
    w, ln = network.synthetic_connectome(N, density, seed=N)
    ln = np.where(ln > 0, np.maximum(ln, 16.0), 0.0)   # delays of 40 steps and more at 4 mm/ms
    conn = network.Connectivity.from_dense(w, ln)
    rng = np.random.default_rng(N)
    I = 9
    x0 = np.stack([rng.uniform(0.05, 0.3, (I, N)), rng.uniform(-1.5, -0.5, (I, N))], -1)
    target = np.corrcoef(rng.normal(size=(N, 60))).astype(np.float32)
    speed = 16.0 / (0.1 * (2.5 * K)) if near else 4.0
    prob = adjoint.FCFit(conn, 0.1, speed, x0.astype(np.float32), target, 130, checkpoint_every=37)
    prob.adj_k = K
    prob.lognh_g = max(1, int(np.ceil(np.log2(prob.dmax + K))))
    assert prob.adjoint_kernel == 'groups' and (2 * K <= prob.dmin < 3 * K if near else prob.dmin >= 3 * K)
    consts = np.array(prob.consts, np.float32)
    consts[2] = tau
    prob.consts = consts
    prob.adjoint_shape = adjoint.adjoint_group_shape(N, pipelined=pipe, slots=8 if N == 41 else 32)
    prob.forward(np.linspace(0.1, 0.5, I).astype(np.float32), rng.uniform(-6, -4, (I, N)).astype(np.float32))
    dG_g, deta_g = (t.clone() for t in prob.backward())
    prob.adjoint_kernel = 'instances'
    dG_i, deta_i = prob.backward()
    assert torch.equal(dG_g, dG_i) and torch.equal(deta_g, deta_i)
    assert bool(torch.isfinite(dG_g).all()) and float(deta_g.abs().max()) > 0
