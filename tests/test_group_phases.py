"""
The pipelined group kernel's phases across the CTAs of a cluster
(run_group_pipelined, csrc/tvbg_lanes.cuh).

Host: with every delay >= 3K - 1 a phase may start when the phase before the
last one is complete everywhere, so one CTA can be a phase ahead of another;
simulated with two CTAs (even and odd nodes) over a modular ring, either of
them ahead, against the step-by-step recursion, and with each condition
broken once.  GPU: the new branches against the oracle at 1e-4 (the
tolerance of every state comparison): phases awaited a phase late or at once,
staged and unstaged edge records, unaligned rings, every CTA build.
"""

import numpy as np
import pytest

from test_group_blocking_host import differs, problem, step_by_step

TOL = 1e-4


def two_ctas(edges, g, x0, K, nh, ahead, a=0.5):
    """CTA `ahead` runs each phase one phase earlier than the other: its
    gather of block b + 2 and its update of block b + 1 see the ring before
    the other CTA's phase b has run, and the other one sees its writes early."""
    T, N = g.shape
    ring = np.zeros((N, nh))
    ring[:, 0] = x0
    x = x0.copy()
    starts = list(range(0, T, K))
    sums = [{}, {}]

    def gather(c, b):
        if b >= len(starts):
            return
        for t in range(starts[b], min(T, starts[b] + K)):
            s = np.zeros(N)
            for j, i, d, w in edges:
                if j % 2 == c:
                    s[j] += w * ring[i, (t - d) % nh]
            sums[c][t] = s

    def phase(c, b):     # update of block b and gather of block b + 1
        gather(c, b + 1)
        own = np.arange(N) % 2 == c
        for t in range(starts[b], min(T, starts[b] + K)):
            x[own] = (a * x + sums[c][t] + g[t])[own]
            ring[own, (t + 1) % nh] = x[own]

    for c in (0, 1):
        gather(c, 0)
    phase(ahead, 0)
    for b in range(len(starts)):
        if b + 1 < len(starts):
            phase(ahead, b + 1)
        phase(1 - ahead, b)
    return x


@pytest.mark.parametrize('ahead', [0, 1])
def test_one_phase_ahead(ahead):
    K = 8
    for seed in range(3):
        edges, g, x0 = problem(dmin=3 * K - 1, dmax=40, seed=seed)
        ref = step_by_step(edges, g, x0)
        assert np.array_equal(two_ctas(edges, g, x0, K, 49, ahead), ref)   # nh = d_max + 1 + K
    edges, g, x0 = problem(dmin=2 * K - 1, dmax=40, seed=3)                # a delay below 3K - 1
    assert differs(two_ctas(edges, g, x0, K, 64, ahead), step_by_step(edges, g, x0))
    edges, g, x0 = problem(dmin=3 * K - 1, dmax=40, seed=4)                # a ring too short
    assert differs(two_ctas(edges, g, x0, K, 41, ahead), step_by_step(edges, g, x0))


# N, density, speed (delays 10-200 mm / speed / 0.1 ms), threads, cluster, tpn
FORMS = [
    (33, 0.9, 6.5, 192, 4, 2),     # d_min 16: every phase awaited at once
    (33, 0.9, 4.0, 192, 4, 2),     # d_min 26: awaited a phase late
    (70, 0.9, 4.0, 576, 2, 2),     # 62 in-edges a node: records read from global memory
    (70, 0.9, 4.0, 576, 1, 1),
    (41, 0.5, 4.0, 704, 1, 2),     # 768-thread build, one CTA
    (57, 0.4, 4.0, 960, 1, 2),     # 1024-thread build
    (100, 0.2, 4.0, 800, 1, 1),    # plain, 1024-thread build
    (17, 0.5, 12.0, 64, 3, 1),     # K = 8, plain cluster
    (17, 0.5, 18.0, 160, 1, 1),    # K = 4
    (8, 0.9, 4.0, 64, 3, 2),       # slots without a node
]


@pytest.mark.gpu
@pytest.mark.parametrize('N,density,speed,threads,cluster,tpn', FORMS)
@pytest.mark.parametrize('pair', [('MPR', 'Linear'), ('Kuramoto', 'Kuramoto')])
def test_forms_against_oracle(cuda, N, density, speed, threads, cluster, tpn, pair):
    import pyoracle as orc
    from conftest import circ_rel_err, rel_err
    gs, x0 = _set(N, density, speed, pair)
    gs.set_shape(threads, cluster, 0, tpn)
    for n in (83, 60):             # a partial last block, then an unaligned start
        gs.run(n)
    err = circ_rel_err if pair[0] == 'Kuramoto' else rel_err
    ref = orc.run_groups_like(gs, x0, 143)
    assert err(gs.state.cpu().numpy(), ref['state']) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize('tpn,offset', [(1, 1), (1, 2), (1, 4), (2, 4)])
@pytest.mark.parametrize('pair', [('MPR', 'Linear'), ('Kuramoto', 'Kuramoto')])
def test_unaligned_ring(cuda, tpn, offset, pair):
    "A ring off the 32-byte boundary (4-byte aligned; 16 for the pipelined kernel): the same bits."
    torch = cuda
    a, _ = _set(30, 0.4, 4.0, pair)
    b, _ = _set(30, 0.4, 4.0, pair)
    big = torch.zeros(b.ring.numel() + offset, device='cuda')
    big[offset:] = b.ring
    b.ring = big[offset:]
    for s in (a, b):
        s.set_shape(*((256, 1, 0, 1) if tpn == 1 else (256, 2, 0, 2)))
        s.run(131)
    assert torch.equal(a.state, b.state) and torch.equal(a.ring, b.ring)


def _set(N, density, speed, pair):
    from tvb_hpc import coupling, groups, model, network, scheme
    w, ln = network.synthetic_connectome(N, density, seed=N)
    conn = network.Connectivity.from_dense(w, ln)
    rng = np.random.default_rng(N)
    m = getattr(model, pair[0])()
    I = 11
    if pair[0] == 'MPR':
        x0 = np.stack([rng.uniform(0.05, 0.3, (I, N)), rng.uniform(-1.5, -0.5, (I, N))], -1)
        p = rng.uniform(-6, -4, (I, N, 1))
    else:
        x0 = rng.uniform(0, 2 * np.pi, (I, N, 1))
        p = rng.normal(0.06, 0.001, (I, N, 1))
    x0 = x0.astype(np.float32)
    gs = groups.GroupSet(m, getattr(coupling, pair[1])(m), scheme.EulerMaryuyamaStep(0.1), conn,
                         dt=0.1, couplings=np.logspace(-2, -1, I).astype(np.float32),
                         speeds=np.full(I, speed, np.float32), state0=x0,
                         nparam=p.astype(np.float32), seed=7)
    return gs, x0
