"""
The executor's packed copies and its ring kernel.  The ring of
tvbg_ring_from_obs against the definition in numpy (bytes equal: it copies
values); a call with numpy arrays, packed or not, against the same call with
CUDA tensors (bytes equal: the same kernels on the same values).
"""

import numpy as np
import pytest

from tvb_hpc import _native as nat
from tvb_hpc import coupling, model, network, scheme, transforms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('I,N,nobs,ntime,lognh,t_lo,rows', [
    (1, 1, 1, 1, 2, 0, 1), (1, 84, 2, 100, 6, -3, 17), (3, 33, 1, 7, 4, -20, 16),
    (2, 68, 2, 50, 5, 93, 32), (4, 5, 3, 11, 3, 10 ** 9 + 7, 0)])
def test_ring(cuda, I, N, nobs, ntime, lognh, t_lo, rows):
    torch = cuda
    nh = 1 << lognh
    ob = np.random.default_rng(N).standard_normal((ntime, I, N, nobs)).astype(np.float32)
    want = np.zeros((I, N, nh), np.float32)
    for t in range(t_lo, t_lo + rows):
        for j in range(N):
            want[:, j, (t + j) % nh] = ob[t % ntime, :, j, 0]
    d = torch.from_numpy(ob).cuda()
    ring = torch.full((I, N * nh), float('nan'), device='cuda')
    nat.check(nat.load().tvbg_ring_from_obs(d.data_ptr(), ntime, I, N, nobs, t_lo, t_lo + rows, lognh,
                                            ring.data_ptr(), nat.stream_handle()))
    assert ring.cpu().numpy().tobytes() == want.tobytes()


@pytest.mark.parametrize('order', ['tracka', 'cuda'])
@pytest.mark.parametrize('I,N,dt,extra', [
    (None, 1, np.float32, 5), (None, 84, np.float64, 40), (3, 33, np.float32, 11),
    (2, 68, np.float32, 2200)])       # the last one is above PACK_BYTES
def test_packed_call(cuda, order, I, N, dt, extra):
    torch = cuda
    rng = np.random.default_rng(7)
    w, ln = network.synthetic_connectome(N, 0.3, seed=3) if N > 1 else (np.zeros((1, 1)), np.zeros((1, 1)))
    c = network.Connectivity.from_dense(w, ln)
    m = model.Kuramoto()
    m.dt = 0.1
    knl = transforms.network_time_step(m, coupling.Kuramoto(m), scheme.EulerStep(0.1), order=order)
    d = c.delays(5.0, 0.1, 'ceil').astype(np.uintc)
    lead = () if I is None else (I, )
    ntime = (int(d.max()) if d.size else 0) + extra
    st = rng.uniform(0, 6, lead + (N, 1)).astype(dt)
    ob = rng.uniform(0, 6, (ntime, ) + lead + (N, 2)).astype(dt)
    pa = np.full((N, 1), 0.06, dt)
    if N == 33:
        st, ob = np.asfortranarray(st), np.asfortranarray(ob)
    small = 4 * (st.size + ob.size + pa.size) + 8 * d.size <= transforms.PACK_BYTES
    assert small == (extra != 2200)
    dev = [torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda() for x in (st, ob, pa)]
    for i in range(3):
        for s, o, p in ((st, ob, pa), (dev[0], dev[1], dev[2])):
            knl(nstep=4, nnode=N, ntime=ntime, state=s, input=None, param=p, drift=None, diffs=None,
                obsrv=o, nnz=c.nnz, delays=d, row=c.row, col=c.col, weights=c.wnz, i_step_0=ntime - 6 + 4 * i)
        assert np.ascontiguousarray(st, np.float32).tobytes() == dev[0].cpu().numpy().tobytes()
        assert np.ascontiguousarray(ob, np.float32).tobytes() == dev[1].cpu().numpy().tobytes()
