"""
Persistent batches (tvbg_batch_run) whose CTAs take several instances in turn,
with rings staged in shared memory that the kernel itself rewrites (Sigmoidal:
the staged ring holds pre(x)): state and ring bit-identical to one instance
per CTA (tvbg_sweep), and equal to rings in global memory up to the rounding
of pre (two ulps of a coupling below 0.01, 96 steps: 1e-5 of the state).
"""

import numpy as np
import pytest

from conftest import rel_err

from tvb_hpc import model, coupling, scheme, network, engine, _native as nat

pytestmark = pytest.mark.gpu


def make(N, I, speed, seed, staged=True):
    w, ln = network.synthetic_connectome(N, 0.3, seed=seed)
    conn = network.Connectivity.from_dense(w, ln)
    m = model.G2DO()
    cf = coupling.Sigmoidal(m)
    x0 = np.random.default_rng(seed).uniform(-0.5, 0.5, (I, N, 2)).astype(np.float32)
    s = engine.Sweep(m, cf, scheme.EulerMaryuyamaStep(0.1), conn, dt=0.1, couplings=np.logspace(-2, 0, I),
                     speeds=speed, state0=x0, seed=11 + seed, tpn=4, history='fill')
    if not staged:
        s.smem_cap = 0
    return s


# 68 nodes at 4 m/s: more than half the shared memory, one CTA per SM; 40 nodes at
# 20 m/s: several CTAs per SM, 4 or 8 steps per block
@pytest.mark.parametrize('sizes', [[(68, 400, 4.0)], [(40, 2000, 20.0)], [(68, 200, 4.0), (84, 200, 6.0)]])
def test_sigmoidal_instances_in_turn(cuda, sizes):
    nsteps = 96
    sets = [make(N, I, v, k) for k, (N, I, v) in enumerate(sizes)]
    batch = engine.Batch(sets, [nsteps] * len(sets), tpn=4)
    assert any(L['n'] > L['cfg'].ctas for L in batch.launches)     # CTAs with a second instance
    for s in sets:
        assert np.all(s.build_table(1)['flags'] & nat.F_SMEM_RING) and np.all(s.block_k > 0)
    batch.run()
    for k, (N, I, v) in enumerate(sizes):
        one = make(N, I, v, k)
        one.run(nsteps)
        assert np.array_equal(sets[k].state.cpu().numpy(), one.state.cpu().numpy())
        assert np.array_equal(sets[k].ring.cpu().numpy(), one.ring.cpu().numpy())
        far = make(N, I, v, k, staged=False)
        assert not np.any(far.build_table(1)['flags'] & nat.F_SMEM_RING)
        far.run(nsteps)
        assert rel_err(one.state.cpu().numpy(), far.state.cpu().numpy()) < 1e-5
        assert rel_err(one.ring.cpu().numpy(), far.ring.cpu().numpy()) < 1e-5
