"""
A gradient request's footprint (serve.fit_bytes) against what FCFit allocates
where it keeps the whole trace: never less (beyond the allocator's rounding and
the tables, 8 MB) and not half as much again, so that the server neither runs
out of memory nor turns away what fits.
"""

import numpy as np
import pytest

from tvb_hpc import adjoint, network, serve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N,I,T,speed', [(84, 64, 1500, 4.0), (68, 200, 400, 4.0), (131, 9, 2000, 6.0),
                                         (400, 8, 500, 4.0)])
def test_fit_bytes(cuda, N, I, T, speed):
    torch = cuda
    w, ln = network.synthetic_connectome(N, 0.2, seed=N)
    conn = network.Connectivity.from_dense(w, ln)
    rng = np.random.default_rng(N)
    x0 = np.stack([rng.uniform(0.05, 0.3, (I, N)), rng.uniform(-1.5, -0.5, (I, N))], -1)
    req = serve.Request(rid=0, model='MPR', conn=conn, couplings=np.full(I, 0.05, np.float32),
                        speeds=np.full(I, speed, np.float32), x0=x0.astype(np.float32), nsteps=T)
    base = serve.footprint(req)
    req.want_grad, req.target = True, np.corrcoef(rng.normal(size=(N, 40)))
    est = serve.footprint(req) - base
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    held = torch.cuda.memory_allocated()
    fit = adjoint.FCFit(conn, 0.1, speed, req.x0, req.target, T)
    fit.forward(req.couplings, rng.uniform(-6, -4, (I, N)).astype(np.float32))
    fit.backward()
    fit.check()
    torch.cuda.synchronize()
    peak = torch.cuda.max_memory_allocated() - held
    assert peak < est + (8 << 20)
    assert fit.layout == 'groups' and fit._traced()
    assert est < 1.5 * peak + (8 << 20)
