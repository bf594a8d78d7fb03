"""
Several blocks of 8 steps per launch (tvbg_net_run_ex) against the one-block
kernels: the same bits, for 2 and 3 blocks, every remainder of steps, delays at
the limits (7, 15, 23 and nh - 9), nodes without edges, and the tail of the
last CTA.
"""

import numpy as np
import pytest

from tvb_hpc import bignet, coupling, model, network, scheme

pytestmark = pytest.mark.gpu


def make(name, cfun_name, N, dmin, dmax, noise, **kw):
    conn = network.synthetic_sparse_connectome(N, 9, seed=N)
    rng = np.random.default_rng(N)
    d = rng.integers(dmin, dmax + 1, conn.col.size).astype(np.int32)
    d[:2] = dmin, dmax
    m = getattr(model, name)()
    x0 = rng.uniform(-0.5, 0.5, (N, m.nsvar)).astype(np.float32)
    return bignet.SingleNetwork(m, getattr(coupling, cfun_name)(m),
                                scheme.EulerMaryuyamaStep(0.1) if noise else scheme.EulerStep(0.1),
                                conn, 0.1, coupling=0.05, delays=d, state0=np.abs(x0), seed=5,
                                block_k=8, **kw)


@pytest.mark.parametrize('name,cfun_name,noise', [('Generic2dOscillator', 'Linear', False),
                                                  ('MPR', 'Diff', True), ('Linear', 'Sigmoidal', True)])
@pytest.mark.parametrize('N,dmin,dmax', [(33, 14, 60), (63, 15, 55), (2049, 23, 119), (500, 40, 503),
                                         (100, 22, 23)])
@pytest.mark.parametrize('steps', [(50, 24, 9, 8, 1), (17, 16, 7, 33)])
def test_same_bits(cuda, name, cfun_name, noise, N, dmin, dmax, steps):
    a = make(name, cfun_name, N, dmin, dmax, noise)
    b = make(name, cfun_name, N, dmin, dmax, noise, lanes=False)   # one thread per node, one block
    assert (a._stage is None) == (dmin < 15) and b._stage is None
    for n in steps:
        a.run(n)
        b.run(n)
    assert np.array_equal(a.state.cpu().numpy(), b.state.cpu().numpy())
    assert np.array_equal(a.ring_plain(), b.ring_plain())
    assert np.array_equal(a.ring.cpu().numpy(), b.ring.cpu().numpy())   # the mirrored slots too
