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


def test_cta_width_follows_the_ring_of_each_launch(cuda):
    """Rings of 64 and 512 slots in one sweep: the launch whose staged ring leaves one
    CTA per SM has 512 threads, the one whose CTAs share an SM 256; the results are those of one speed at
    a time."""
    speeds = [4.0, 40.0]
    w, ln = network.synthetic_connectome(68, 0.3, seed=0)
    conn = network.Connectivity.from_dense(w, ln)
    m = model.MPR()
    x0 = np.random.default_rng(1).uniform(0.05, 0.3, (6, 68, 2)).astype(np.float32)

    def sweep(v, ids):
        return engine.Sweep(m, coupling.Linear(m), scheme.EulerMaryuyamaStep(0.1), conn, dt=0.1,
                            couplings=np.full(len(ids), 0.1), speeds=np.asarray(v, np.float32),
                            state0=x0[ids], seed=5, tpn=4, inst_ids=ids)

    s = sweep(np.resize(speeds, 6), np.arange(6))
    width = {}
    for _, _, smem, bk in s.prepare(40):
        assert smem > 0 and bk > 0
        width[2 * smem > s.smem_cap] = s._launch_cfg(smem, 4, bk).threads
    assert width == {True: 512, False: 256}
    s.run(40)
    for k, v in enumerate(speeds):
        ids = np.arange(k, 6, 2)
        one = sweep([v] * 3, ids)
        one.run(40)
        assert np.array_equal(s.state.cpu().numpy()[ids], one.state.cpu().numpy())
