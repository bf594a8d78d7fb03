"""
Two host threads that launch one kernel with CTAs of different shared memory,
each on a stream of its own: no launch is refused (a kernel's opt-in limit
belongs to the kernel, so a thread that sets it to its own size takes it from
the other between that one's call and its launch), and the results stay those
of one thread.
"""

import ctypes
import threading

import numpy as np
import pytest

from tvb_hpc import model, coupling, scheme, network, groups, _native as nat

pytestmark = pytest.mark.gpu

CALLS = 3000


def group_calls(torch, N, threads, tpn):
    w, ln = network.synthetic_connectome(N, 0.1, seed=N)
    conn = network.Connectivity.from_dense(w, ln)
    m = model.MPR()
    x0 = np.random.default_rng(N).uniform(0.05, 0.3, (8, N, 2)).astype(np.float32)
    s = groups.GroupSet(m, coupling.Linear(m), scheme.EulerStep(0.1), conn, dt=0.1, couplings=np.full(8, 0.1),
                        speeds=2.0, state0=x0)
    s.set_shape(threads, 1, 0, tpn)
    launches = s.prepare_segments([(0, 8)])[0]
    (dev, order, n, cfg), = launches
    fn = nat.load().tvbg_group_run
    return (lambda h: fn(dev.data_ptr(), n, ctypes.byref(cfg), h)), (s, launches)


def rmap_calls(torch, nroi):
    n = 4096
    rmap = torch.arange(n, dtype=torch.int32, device='cuda') % nroi
    node = torch.ones(n, 1, device='cuda')
    roi = torch.empty(nroi, 1, device='cuda')
    fn = nat.load().tvbg_rmap_to_avg
    return (lambda h: fn(nroi, 1, n, rmap.data_ptr(), node.data_ptr(), roi.data_ptr(), h)), (rmap, node, roi)


def cov_calls(torch, N, rows):
    x = torch.ones(1, rows, N, device='cuda')
    mean = torch.zeros(1, N, dtype=torch.float64, device='cuda')
    m2 = torch.zeros(1, N, N, dtype=torch.float64, device='cuda')
    fn = nat.load().tvbg_cov_update_rows
    return (lambda h: fn(x.data_ptr(), rows * N, N, rows, 1, N, 0, mean.data_ptr(), m2.data_ptr(), h)), (x, mean, m2)


def fc_calls(torch, N):
    x = torch.rand(1, 20, N, device='cuda')
    fc = torch.empty(1, N, N, device='cuda')
    fn = nat.load().tvbg_fc
    return (lambda h: fn(x.data_ptr(), 1, 20, N, 20 * N, fc.data_ptr(), None, None, h)), (x, fc)


PAIRS = {
    'group': (group_calls, (80, 640, 1), (96, 768, 1)),
    'pipelined': (group_calls, (56, 896, 2), (64, 1024, 2)),
    'rmap': (rmap_calls, (68, ), (1600, )),
    'cov': (cov_calls, (340, 9), (500, 16)),
    'fc': (fc_calls, (20, ), (96, )),
}


@pytest.mark.parametrize('kind', sorted(PAIRS))
def test_two_threads(cuda, kind):
    torch = cuda
    make, a, b = PAIRS[kind]
    calls = [make(torch, *a), make(torch, *b)]
    streams = [torch.cuda.Stream() for _ in calls]
    for (fn, _), s in zip(calls, streams):     # module loading
        nat.check(fn(s.cuda_stream))
    torch.cuda.synchronize()
    refused = [0, 0]
    gate = threading.Barrier(2)

    def work(k):
        fn, h = calls[k][0], streams[k].cuda_stream
        gate.wait()
        for _ in range(CALLS):
            refused[k] += fn(h) != 0

    ts = [threading.Thread(target=work, args=(k, )) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert refused == [0, 0]
