"""
Performance cases of the engine: what its users run, through the public
entry points, from one drop-in step call to whole parameter sweeps, an uneven
batch, one very large network, FC-fit gradients and the metrics after a run.

Every pass starts from the initial state it was given (the state is reset
inside the pass, as a program that runs one sweep after another does), so a
pass can be repeated and its outputs depend on the inputs alone.  ``exact``
restates each computation in 64 bits with plain torch.
"""

import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, 'tvb-hpc_gb300') not in sys.path:
    sys.path.insert(1, os.path.join(ROOT, 'tvb-hpc_gb300'))

from tvb_hpc import (  # noqa: E402
    adjoint, bignet, coupling, engine, groups, lems, metric, model, network, scheme, transforms)

F64 = torch.float64
DT = 0.1                      # ms, every sweep
LEN_LO, LEN_HI = 10.0, 200.0  # mm, tract lengths of the synthetic connectomes


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the drop-in executor as the hackathon driver calls it: ten steps of
        # one 84-node Kuramoto network with numpy arrays -- the smallest call
        dict(name='step_call_84', kind='step', N=84, subjects=1, nstep=10),
        # the parity configuration: 32 couplings of a 68-node Kuramoto network
        dict(name='sweep_kuramoto_32', kind='sweep', model='Kuramoto', cfun='Kuramoto', N=68,
             density=0.30, I=32, nsteps=1000, speed_lo=4.0, speed_hi=4.0, n_speeds=1, noise=False,
             bold=0, prepared=False),
        # the 64 x 64 coupling x speed grid with BOLD and FC (speeds 1-20
        # mm/ms: long and short delays), tables prepared once: the largest sweep
        dict(name='sweep_grid_4096_bold_fc', kind='sweep', model='Generic2dOscillator', cfun='Diff',
             N=84, density=0.30, I=4096, nsteps=2000, speed_lo=1.0, speed_hi=20.0, n_speeds=64,
             noise=True, bold=50, prepared=True),
        # an exploratory sweep of odd size: 77 points of a 131-node stochastic
        # mean-field network, one simple run() call
        dict(name='sweep_mpr_77x131', kind='sweep', model='MPR', cfun='Linear', N=131, density=0.20,
             I=77, nsteps=1500, speed_lo=4.0, speed_hi=4.0, n_speeds=1, noise=True, bold=0,
             prepared=False),
        # the uneven batch: five connectomes of 68-998 nodes with uneven step
        # counts, launch shapes tuned, captured into one graph
        dict(name='batch_uneven_5', kind='batch', nodes='68,84,192,400,998',
             densities='0.30,0.30,0.15,0.08,0.03', instances='1024,1024,256,64,16',
             steps_lo=500, steps_hi=5000),
        # engine.Sweep, the per-instance path, on a sigmoidal coupling
        dict(name='instances_sigmoidal_200', kind='instances', model='Generic2dOscillator',
             cfun='Sigmoidal', N=84, density=0.30, I=200, nsteps=500, speed=4.0, noise=True),
        # the DSL's default 32 x 32 sweep on a model generated from LEMS XML
        dict(name='lems_epileptor_1024', kind='lems', N=68, density=0.30, n_speeds=32, n_couplings=32,
             nsteps=400),
        # one simulation of the 515 056-node network
        dict(name='net_515056', kind='net', N=515056, degree=64, nsteps=96),
        # gradients of an FC fit: forward and adjoint of 256 instances
        dict(name='fcfit_256x84', kind='adjoint', N=84, density=0.30, I=256, T=2000, ckpt=100),
        # Pearson FC of finished series with the fit error, nodes beyond the
        # one-CTA size
        dict(name='fc_16x400', kind='fc', I=16, T=1200, N=400),
        # streaming FC of a running sweep: eight new BOLD rows, then the FC
        dict(name='streaming_fc_256x84', kind='stream', I=256, N=84, rows=8),
        # region averages of a cortical surface (two variables) and back
        dict(name='region_map_515056', kind='rmap', nnode=515056, nroi=68, nvar=2),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _density(N):
    "Connectome density by size: 30 % up to 84 nodes, 3 % at 998 (the benchmark's batch)."
    return round(min(0.30, max(0.03, 0.30 * (84.0 / N) ** 0.93)), 3)


def draw(rng):
    kind = rng.choice(['step', 'sweep', 'sweep', 'sweep', 'batch', 'instances', 'lems', 'net',
                       'adjoint', 'fc', 'stream', 'rmap'])
    if kind == 'step':
        return dict(kind=kind, N=_logint(rng, 20, 400), subjects=_logint(rng, 1, 16),
                    nstep=_logint(rng, 1, 64))
    if kind == 'sweep':
        mod, cf = rng.choice([('Kuramoto', 'Kuramoto'), ('Generic2dOscillator', 'Diff'),
                              ('MPR', 'Linear'), ('MPR', 'Diff'), ('RWW', 'Linear'),
                              ('Generic2dOscillator', 'Sigmoidal')])
        N = _logint(rng, 20, 700)
        nsteps = _logint(rng, 100, 3000)
        I = _logint(rng, 1, max(8, min(4096, int(2e8 / (N * nsteps)))))
        lo = rng.choice([2.0, 4.0, 6.0])
        many = rng.random() < 0.4 and I >= 16
        return dict(kind=kind, model=mod, cfun=cf, N=N, density=_density(N), I=I, nsteps=nsteps,
                    speed_lo=lo, speed_hi=rng.choice([12.0, 20.0]) if many else lo,
                    n_speeds=rng.randint(2, 8) if many else 1, noise=rng.random() < 0.7,
                    bold=rng.choice([0, 0, max(5, nsteps // 40)]), prepared=rng.random() < 0.5)
    if kind == 'batch':
        k = rng.randint(2, 5)
        nodes = sorted(_logint(rng, 30, 998) for _ in range(k))
        inst = [max(1, int(rng.uniform(0.2, 0.8) * min(1024, 60000 // n))) for n in nodes]
        lo = _logint(rng, 100, 500)
        return dict(kind=kind, nodes=','.join(map(str, nodes)),
                    densities=','.join(str(_density(n)) for n in nodes),
                    instances=','.join(map(str, inst)), steps_lo=lo, steps_hi=lo * rng.randint(2, 6))
    if kind == 'instances':
        mod, cf = rng.choice([('Generic2dOscillator', 'Sigmoidal'), ('RWW', 'Linear'),
                              ('MPR', 'Diff'), ('Kuramoto', 'Kuramoto')])
        N = _logint(rng, 20, 400)
        return dict(kind=kind, model=mod, cfun=cf, N=N, density=_density(N),
                    I=_logint(rng, 1, 300), nsteps=_logint(rng, 50, 800),
                    speed=rng.choice([4.0, 8.0]), noise=rng.random() < 0.6)
    if kind == 'lems':
        N = _logint(rng, 30, 200)
        return dict(kind=kind, N=N, density=_density(N), n_speeds=rng.randint(2, 32),
                    n_couplings=rng.randint(4, 32), nsteps=_logint(rng, 50, 400))
    if kind == 'net':
        return dict(kind=kind, N=_logint(rng, 10000, 515056), degree=rng.randint(16, 64),
                    nsteps=_logint(rng, 16, 96))
    if kind == 'adjoint':
        N = _logint(rng, 30, 150)
        return dict(kind=kind, N=N, density=_density(N), I=_logint(rng, 4, 200),
                    T=100 * rng.randint(2, 18) + rng.randint(0, 99), ckpt=rng.choice([50, 100]))
    if kind == 'fc':
        N = _logint(rng, 30, 500)
        return dict(kind=kind, I=_logint(rng, 1, 64), T=_logint(rng, 50, 1500), N=N)
    if kind == 'stream':
        N = _logint(rng, 30, 400)
        return dict(kind=kind, I=_logint(rng, 1, max(2, min(512, int(8e6 / (N * N))))), N=N,
                    rows=rng.randint(1, 12))
    return dict(kind=kind, nnode=_logint(rng, 5000, 515056), nroi=_logint(rng, 16, 400),
                nvar=rng.randint(1, 4))


# ---------------------------------------------------------------------------
# inputs (shared by prepare and exact)
# ---------------------------------------------------------------------------
def _conn(N, density, seed):
    w, ln = network.synthetic_connectome(N, density, seed=seed, len_lo=LEN_LO, len_hi=LEN_HI)
    return network.Connectivity.from_dense(w, ln)


def _start(name, rng, I, N):
    "Initial state and per-node parameters of a sweep."
    if name == 'Kuramoto':
        return (rng.uniform(0, 2 * np.pi, (I, N, 1)).astype(np.float32),
                rng.normal(2 * np.pi * 0.01, 0.001, (I, N, 1)).astype(np.float32))
    if name == 'MPR':
        x = np.stack([rng.uniform(0.05, 0.3, (I, N)), rng.uniform(-1.5, -0.5, (I, N))], -1)
        return x.astype(np.float32), rng.uniform(-6, -4, (I, N, 1)).astype(np.float32)
    if name == 'RWW':
        return (rng.uniform(0.1, 0.3, (I, N, 1)).astype(np.float32),
                np.stack([rng.uniform(0.5, 0.7, (I, N)), rng.uniform(0.3, 0.34, (I, N))],
                         -1).astype(np.float32))
    return (rng.uniform(-0.5, 0.5, (I, N, 2)).astype(np.float32),
            rng.uniform(-2.2, -1.8, (I, N, 1)).astype(np.float32))


def _coupling_range(name, I):
    lo, hi = {'Kuramoto': (-2, 1), 'MPR': (-2, -0.5), 'RWW': (-3, -1)}.get(name, (-3, 0))
    return np.logspace(lo, hi, I).astype(np.float32)


def _sweep_inputs(c, seed):
    rng = np.random.default_rng(seed)
    conn = _conn(c['N'], c['density'], seed)
    I = c['I']
    x0, par = _start(c['model'], rng, I, c['N'])
    if c['kind'] == 'instances':
        sp = np.full(I, c['speed'], np.float32)
        a = _coupling_range(c['model'], I)
    else:
        ns = min(c['n_speeds'], I)
        na = -(-I // ns)
        a = np.repeat(_coupling_range(c['model'], na), ns)[:I]
        sp = np.tile(np.linspace(c['speed_lo'], c['speed_hi'], ns).astype(np.float32), na)[:I]
    target = np.corrcoef(rng.normal(size=(c['N'], 200))).astype(np.float32)
    return conn, x0, par, a, sp, target


def _batch_parts(c, seed):
    parts = []
    for k, (N, dens, I) in enumerate(zip(c['nodes'].split(','), c['densities'].split(','),
                                         c['instances'].split(','))):
        N, I = int(N), int(I)
        rng = np.random.default_rng(1000 * seed + k)
        x0, eta = _start('MPR', rng, I, N)
        parts.append((_conn(N, float(dens), 1000 * seed + k), x0, eta, _coupling_range('MPR', I),
                      rng.integers(c['steps_lo'], c['steps_hi'] + 1, I), seed + k))
    return parts


def _step_inputs(c, seed):
    rng = np.random.default_rng(seed)
    N, S = c['N'], c['subjects']
    conn = _conn(N, _density(N), seed)
    lnz = network.delays_f32(conn.lnz, 4.0, 1.0, 'trunc').astype(np.uintc)
    ntime = 1 << int(lnz.max() + c['nstep'] + 1).bit_length()
    th = rng.uniform(0, 2 * np.pi, (S, N, 1)).astype(np.float32)
    par = rng.normal(2 * np.pi * 0.01, 0.001, (S, N, 1)).astype(np.float32)
    obs = rng.uniform(0, 2 * np.pi, (ntime, S, N, 2)).astype(np.float32)
    obs[..., 1] = np.sin(obs[..., 0])
    a = np.logspace(-1, 0, S).astype(np.float32)
    if S == 1:
        return conn, lnz, ntime, th[0], par[0], obs[:, 0], float(a[0])
    return conn, lnz, ntime, th, par, obs, a


def _lems_inputs(c, seed):
    rng = np.random.default_rng(seed)
    conn = _conn(c['N'], c['density'], seed)
    sp = np.logspace(0.0, 2.0, c['n_speeds'])
    cp = np.logspace(-2.0, 0.0, c['n_couplings'])
    params = np.stack(np.meshgrid(sp, cp, indexing='ij'), -1).reshape(-1, 2).astype(np.float32)
    x0 = np.zeros((params.shape[0], c['N'], 6), np.float32)
    for v, (lo, hi) in enumerate([(-1.8, -1.2), (-15, -12), (2.8, 3.2), (-1.2, -0.8), (0, 0.2),
                                  (-0.1, 0.1)]):
        x0[:, :, v] = rng.uniform(lo, hi, x0.shape[:2])
    return conn, params, x0


def _net_inputs(c, seed):
    "Sparse in-edges: Poisson(degree) distinct sources per node, columns sorted in each row."
    N = c['N']
    g = torch.Generator('cuda').manual_seed(seed)
    deg = torch.poisson(torch.full((N, ), float(c['degree']), device='cuda'), generator=g).long()
    tgt = torch.repeat_interleave(torch.arange(N, device='cuda'), deg)
    src = torch.randint(0, N, (tgt.numel(), ), generator=g, device='cuda')
    key = torch.unique(tgt * N + src)
    tgt, src = key // N, key % N
    row = torch.zeros(N + 1, dtype=torch.int64, device='cuda')
    row[1:] = torch.cumsum(torch.bincount(tgt, minlength=N), 0)
    nnz = int(src.numel())
    w = torch.randn(nnz, generator=g, device='cuda').sub_(1.0).exp_()
    w = w / w.max()
    ln = torch.rand(nnz, generator=g, device='cuda') * (LEN_HI - LEN_LO) + LEN_LO
    conn = network.Connectivity(N, None, nnz, src.int().cpu().numpy(), row.int().cpu().numpy(),
                                w.cpu().numpy(), ln.cpu().numpy())
    x0 = (torch.rand((N, 2), generator=g, device='cuda') - 0.5).cpu().numpy()
    return conn, x0


def _fit_inputs(c, seed):
    rng = np.random.default_rng(seed)
    conn = _conn(c['N'], c['density'], seed)
    x0, eta = _start('MPR', rng, c['I'], c['N'])
    target = np.corrcoef(rng.normal(size=(c['N'], 60))).astype(np.float32)
    return conn, x0, eta[:, :, 0], _coupling_range('MPR', c['I']), target


def _series(I, T, N, seed):
    "Slow correlated series around a baseline, as BOLD rows are."
    g = torch.Generator('cuda').manual_seed(seed)
    mix = torch.randn((I, N, 8), generator=g, device='cuda')
    common = torch.cumsum(torch.randn((I, T, 8), generator=g, device='cuda'), 1) * 0.1
    own = torch.randn((I, T, N), generator=g, device='cuda')
    return (1.0 + 0.02 * (common @ mix.transpose(1, 2) + own)).float().contiguous()


def _target(N, seed):
    rng = np.random.default_rng(seed)
    return np.corrcoef(rng.normal(size=(N, 200))).astype(np.float32)


def _rmap_inputs(c, seed):
    g = torch.Generator('cuda').manual_seed(seed)
    rmap = torch.sort(torch.randint(0, c['nroi'], (c['nnode'], ), generator=g, device='cuda',
                                    dtype=torch.int32))[0]
    # regions are contiguous patches of the surface's node order, ragged in size
    node = torch.randn((c['nnode'], c['nvar']), generator=g, device='cuda')
    return rmap.contiguous(), node


def _make(name, cfname):
    m = getattr(model, name)()
    return m, getattr(coupling, cfname)(m)


def _scheme(noise):
    return scheme.EulerMaryuyamaStep(DT) if noise else scheme.EulerStep(DT)


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    c = case
    kind = c['kind']
    if kind == 'step':
        conn, lnz, ntime, th, par, obs, a = _step_inputs(c, seed)
        osc = model.Kuramoto()
        osc.dt = 1.0
        cf = coupling.Kuramoto(osc)
        cf.param['a'] = 'a'
        knl = transforms.network_time_step(osc, cf, scheme.EulerStep(1.0))
        return dict(c=c, knl=knl, conn=conn, lnz=lnz, ntime=ntime, th=th, par=par, obs=obs, a=a,
                    scratch=[np.zeros(th.shape, np.float32) for _ in range(3)])
    if kind == 'sweep':
        conn, x0, par, a, sp, target = _sweep_inputs(c, seed)
        m, cf = _make(c['model'], c['cfun'])
        s = groups.GroupSet(m, cf, _scheme(c['noise']), conn, dt=DT, couplings=a, speeds=sp,
                            state0=x0, nparam=par, seed=seed, bold_period=c['bold'],
                            bold_len=c['nsteps'] // c['bold'] if c['bold'] else 0)
        st = dict(c=c, s=s, x0=s.state.clone(), target=torch.from_numpy(target).cuda())
        if c['prepared']:
            st['launches'] = s.prepare(c['nsteps'])[0]
        return st
    if kind == 'batch':
        m, cf = _make('MPR', 'Linear')
        parts = _batch_parts(c, seed)
        sets = [groups.GroupSet(m, cf, _scheme(True), conn, dt=DT, couplings=a, speeds=4.0,
                                state0=x0, nparam=eta, seed=sd, nsteps=steps)
                for conn, x0, eta, a, steps, sd in parts]
        x0s = [s.state.clone() for s in sets]
        b = groups.GroupBatch(sets, [p[4] for p in parts], shapes='tune')
        b.capture()
        return dict(c=c, b=b, sets=sets, x0=x0s)
    if kind == 'instances':
        conn, x0, par, a, sp, _ = _sweep_inputs(c, seed)
        m, cf = _make(c['model'], c['cfun'])
        s = engine.Sweep(m, cf, _scheme(c['noise']), conn, dt=DT, couplings=a, speeds=sp, state0=x0,
                         nparam=par, seed=seed, tpn=4)
        return dict(c=c, s=s, x0=s.state.clone())
    if kind == 'lems':
        conn, params, x0 = _lems_inputs(c, seed)
        m = lems.load_model('Epileptor')
        s = lems.make_set(m, conn, DT, params, state0=x0, noise=True, single=True, seed=seed)
        return dict(c=c, s=s, x0=s.state.clone())
    if kind == 'net':
        conn, x0 = _net_inputs(c, seed)
        m, cf = _make('Generic2dOscillator', 'Linear')
        s = bignet.SingleNetwork(m, cf, scheme.EulerStep(DT), conn, DT, coupling=0.05, speed=4.0,
                                 state0=x0, seed=seed)
        return dict(c=c, s=s, x0=s.state.clone())
    if kind == 'adjoint':
        conn, x0, eta, G, target = _fit_inputs(c, seed)
        fit = adjoint.FCFit(conn, dt=DT, speed=4.0, x0=x0, target=target, T=c['T'],
                            checkpoint_every=c['ckpt'])
        return dict(c=c, fit=fit, G=G, eta=eta)
    if kind == 'fc':
        return dict(c=c, x=_series(c['I'], c['T'], c['N'], seed),
                    target=torch.from_numpy(_target(c['N'], seed)).cuda())
    if kind == 'stream':
        return dict(c=c, x=_series(c['I'], c['rows'], c['N'], seed))
    rmap, node = _rmap_inputs(c, seed)
    return dict(c=c, rmap=rmap, node=node, to=network.RMapToAvg().kernel(),
                back=network.RMapFromAvg().kernel(),
                roi=torch.empty((c['nroi'], c['nvar']), device='cuda'),
                out=torch.empty_like(node))


def run(state):
    c = state['c']
    kind = c['kind']
    if kind == 'step':
        th, obs = state['th'].copy(), state['obs'].copy()
        conn, (inp, drift, diffs) = state['conn'], state['scratch']
        state['knl'](nstep=c['nstep'], nnode=c['N'], ntime=state['ntime'], state=th, input=inp,
                     param=state['par'], drift=drift, diffs=diffs, obsrv=obs, nnz=int(conn.nnz),
                     delays=state['lnz'], row=conn.row, col=conn.col, weights=conn.wnz,
                     a=state['a'], i_step_0=state['ntime'])
        return [th, obs]
    if kind == 'sweep':
        s = state['s']
        s.reset(state['x0'])
        if c['prepared']:
            s.launch(state['launches'])
        else:
            s.run(c['nsteps'])
        out = [s.state]
        if c['bold']:
            bold = s.bold_out
            out += [bold] + list(metric.fc(bold, state['target']))
        return out
    if kind == 'batch':
        for s, x in zip(state['sets'], state['x0']):
            s.reset(x)
        state['b'].run(check=False)
        return [s.state for s in state['sets']]
    if kind == 'instances':
        s = state['s']
        s.state.copy_(state['x0'])
        s.ring.zero_()
        s.t[:] = 0
        s.run(c['nsteps'])
        return [s.state.clone()]
    if kind == 'lems':
        s = state['s']
        s.reset(state['x0'])
        s.run(c['nsteps'])
        return [s.state, s.exposures()]
    if kind == 'net':
        s = state['s']
        s.state.copy_(state['x0'])
        s.ring.zero_()
        s.t = 0
        s.run(c['nsteps'])
        return [s.state.clone()]
    if kind == 'adjoint':
        loss = state['fit'].forward(state['G'], state['eta'])
        dG, deta = state['fit'].backward()
        return [loss, dG, deta]
    if kind == 'fc':
        return list(metric.fc(state['x'], state['target']))
    if kind == 'stream':
        f = metric.StreamingFC(c['I'], c['N'])
        f.update_rows(state['x'], range(c['rows']))
        return [f.mean, f.m2, f.corr()]
    a = dict(nroi=c['nroi'], nvar=c['nvar'], nnode=c['nnode'], rmap=state['rmap'], roi=state['roi'])
    state['to'](node=state['node'], **a)
    state['back'](node=state['out'], **a)
    return [state['roi'], state['out']]


# ---------------------------------------------------------------------------
# work: inputs read once, outputs written once, and the arithmetic of the step
# ---------------------------------------------------------------------------
_NS = {'Kuramoto': 1, 'RWW': 1, 'MPR': 2, 'Generic2dOscillator': 2}
# drift and Euler step of one node, without noise; a normal costs about 40
_DRIFT = {'Kuramoto': 45, 'RWW': 30, 'MPR': 20, 'Generic2dOscillator': 22}


def _step_flops(name, cfun, degree, noise, bold):
    per_edge = 4 if cfun == 'Kuramoto' else 2
    ns = _NS[name]
    return per_edge * degree + _DRIFT[name] + (42 * ns if noise else 0) + (60 if bold else 0)


def work(case):
    c = case
    kind = c['kind']
    if kind == 'step':
        N, S = c['N'], c['subjects']
        deg = _density(N) * (N - 1)
        return dict(bytes=S * N * 4 * (3 + 3 * c['nstep']) + 12 * deg * N,
                    flops=S * N * c['nstep'] * (45.0 * deg + 25))
    if kind in ('sweep', 'instances'):
        N, I = c['N'], c['I']
        deg = c['density'] * (N - 1)
        bold = c.get('bold', 0)
        rows = c['nsteps'] // bold if bold else 0
        return dict(bytes=I * N * 4 * (2 * _NS[c['model']] + 1 + rows) + I * N * N * (4 if bold else 0)
                    + 8 * deg * N * c.get('n_speeds', 1),
                    flops=float(I) * N * c['nsteps'] *
                    _step_flops(c['model'], c['cfun'], deg, c['noise'], bold) + I * float(rows) * N * N)
    if kind == 'batch':
        b = f = 0.0
        for N, d, I in zip(c['nodes'].split(','), c['densities'].split(','), c['instances'].split(',')):
            N, I, deg = int(N), int(I), float(d) * (int(N) - 1)
            b += I * N * 20.0 + 8 * deg * N
            f += I * N * 0.5 * (c['steps_lo'] + c['steps_hi']) * _step_flops('MPR', 'Linear', deg, True, 0)
        return dict(bytes=b, flops=f)
    if kind == 'lems':
        N, I = c['N'], c['n_speeds'] * c['n_couplings']
        deg = c['density'] * (N - 1)
        return dict(bytes=I * N * 56.0 + 8 * deg * N * c['n_speeds'],
                    flops=float(I) * N * c['nsteps'] * (4 * deg + 110 + 6 * 42))
    if kind == 'net':
        N, E = c['N'], c['N'] * c['degree']
        return dict(bytes=10.0 * E + 20.0 * N, flops=float(c['nsteps']) * (2 * E + 22 * N))
    if kind == 'adjoint':
        N, I, T = c['N'], c['I'], c['T']
        deg = c['density'] * (N - 1)
        fwd = I * float(N) * T * (2 * deg + 20)
        return dict(bytes=I * N * 24.0 + 16 * deg * N + 8 * I * N,
                    flops=2 * fwd + I * float(N) * T * 30 + I * float(T) * N * N * 3)
    if kind == 'fc':
        I, T, N = c['I'], c['T'], c['N']
        return dict(bytes=4.0 * I * (T * N + N * N), flops=float(I) * T * N * (N + 1))
    if kind == 'stream':
        I, N, R = c['I'], c['N'], c['rows']
        return dict(bytes=4.0 * I * N * R + 12.0 * I * N * N, flops=2.0 * I * N * N * R)
    n = c['nnode']
    return dict(bytes=4.0 * n * (1 + 2 * c['nvar']), flops=float(n) * c['nvar'])


# ---------------------------------------------------------------------------
# exact: the same computations in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _philox(c0, c1, c2, c3, k0, k1):
    "Philox4x32-10 words of int64 tensors holding 32-bit counters and keys."
    M = 0xffffffff
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & M) ^ c1 ^ k0, p1 & M, ((p0 >> 32) & M) ^ c3 ^ k1, p0 & M)
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c0, c1, c2, c3


def _normals(N, inst, call, seed, word3=0):
    "Four normals [4, N, I] of counter (node, call), key (seed, instance)."
    n = torch.arange(N, device='cuda')[:, None]
    zero = torch.zeros((N, inst.numel()), dtype=torch.int64, device='cuda')
    w = _philox(zero + n, zero + call, zero + ((seed >> 32) & 0xffffffff), zero + word3,
                zero + (seed & 0xffffffff), zero + inst[None, :])
    out = []
    for a, b in ((w[0], w[1]), (w[2], w[3])):
        u1 = ((a >> 8).to(F64) + 0.5) * 2.0 ** -24
        ang = (b >> 8).to(F64) * (2.0 ** -23 * math.pi)
        r = torch.sqrt(-2.0 * torch.log(u1))
        out += [r * torch.cos(ang), r * torch.sin(ang)]
    return torch.stack(out)


def _f32(v):
    return float(np.float32(v))


def _drift(name, x, cin, p, m):
    k = {n: _f32(v) for n, v in m.const.items()}
    if name == 'Kuramoto':
        return [p[0] + cin]
    if name == 'MPR':
        r, V = x
        return [(k['Delta'] / (math.pi * k['tau']) + 2 * r * V) / k['tau'],
                (V * V + p[0] + k['J'] * k['tau'] * r + k['I'] + cin
                 - (math.pi * k['tau'] * r) ** 2) / k['tau']]
    if name == 'RWW':
        y = k['a'] * (p[0] * k['J'] * x[0] + p[1] + k['J'] * cin) - k['b']
        h = y / (1.0 - torch.exp(-k['d'] * y))
        return [-x[0] / k['ts'] + (1 - x[0]) * h * k['g']]
    V, W = x
    return [k['d'] * k['tau'] * (k['alpha'] * W - k['f'] * V ** 3 + k['e'] * V * V + k['g'] * V
                                 + k['gamma'] * k['I'] + k['gamma'] * cin),
            k['d'] * (p[0] + k['b'] * V + k['c'] * V * V - k['beta'] * W) / k['tau']]


def _wrap(v):
    tp = 2 * math.pi
    return torch.where(v < 0, v + tp, torch.where(v > tp, v - tp, v))


class _History:
    "Delayed coupling sums over in-edges, instances last: hist[slot][node][instance]."

    def __init__(self, conn, delays, N, I):
        # delays: [nnz] or [nnz, I]
        self.N, self.I = N, I
        row = torch.from_numpy(np.asarray(conn.row, np.int64)).cuda()
        self.tgt = torch.repeat_interleave(torch.arange(N, device='cuda'), row[1:] - row[:-1])
        self.col = torch.from_numpy(np.asarray(conn.col, np.int64)).cuda()
        self.w = torch.from_numpy(np.asarray(conn.wnz, np.float32)).cuda().to(F64)[:, None]
        self.d = torch.from_numpy(np.asarray(delays, np.int64)).cuda()
        self.nh = int(self.d.max()) + 2 if self.d.numel() else 2
        self.h = torch.zeros((self.nh, N, I), dtype=F64, device='cuda')
        if self.d.dim() == 2:
            self.lane = torch.arange(I, device='cuda')[None, :]

    def read(self, t):
        slot = torch.remainder(t - self.d, self.nh)
        if self.d.dim() == 1:
            return self.h.view(-1, self.I)[slot * self.N + self.col]
        return self.h.view(-1)[(slot * self.N + self.col[:, None]) * self.I + self.lane]

    def sum(self, v):
        return torch.zeros((self.N, self.I), dtype=F64, device='cuda').index_add_(0, self.tgt, self.w * v)

    def write(self, t, v):
        self.h[t % self.nh] = v


def _balloon(st, x, dt):
    ts, tf, to, al, e0 = 0.65, 0.41, 0.98, 0.32, 0.4
    s, f, v, q = st
    fv = (1 + v) ** (1 / al)
    dv = (f + 1 - fv) / to
    dq = ((1 + f) * (1 - (1 - e0) ** (1 / (1 + f))) / e0 - fv * (1 + q) / (1 + v)) / to
    return [s + dt * (x - s / ts - f / tf), f + dt * s, v + dt * dv, q + dt * dq]


def _bold_signal(v, q):
    te, v0, e0, eps, nu0, r0 = 0.04, 4.0, 0.4, 0.5, 40.3, 25.0
    return v0 * (-4.3 * nu0 * e0 * te * q + eps * r0 * e0 * te * (v - q) / (1 + v) - (1 - eps) * v)


def _simulate(name, cfname, conn, x0, par, a, sp, steps, noise, seed, bold=0):
    "States [I, N, ns] (and BOLD rows) after `steps` ([I] or scalar) steps."
    m, cf = _make(name, cfname)
    I, N, ns = x0.shape
    uniq, tab = np.unique(sp, return_inverse=True)
    D = np.stack([network.delays_f32(conn.lnz, s, DT, 'ceil') for s in uniq], 1)
    H = _History(conn, D[:, 0] if uniq.size == 1 else D[:, tab], N, I)
    dt = _f32(DT)
    sq = float(np.sqrt(np.float32(DT)))
    x = list(torch.from_numpy(x0).cuda().to(F64).permute(2, 1, 0).contiguous())
    p = torch.from_numpy(par).cuda().to(F64).permute(2, 1, 0)
    av = torch.from_numpy(np.asarray(a, np.float32)).cuda().to(F64)[None, :]
    bv = _f32(cf.param.get('b', 0.0))
    sig = [_f32(v) for v in m.engine_spec()[2]]
    noise = noise and any(sig)
    inst = torch.arange(I, device='cuda')
    steps = np.broadcast_to(np.asarray(steps), (I, ))
    last = torch.from_numpy(np.ascontiguousarray(steps)).cuda()
    spc = 4 // ns
    bst = [torch.zeros((N, I), dtype=F64, device='cuda') for _ in range(4)]
    rows = []
    for t in range(int(steps.max())):
        if noise and t % spc == 0:
            z = _normals(N, inst, t // spc, seed)
        H.write(t, x[0])
        v = H.read(t)
        if cfname == 'Kuramoto':
            cin = av * H.sum(torch.sin(v - x[0][H.tgt])) / N
        elif cfname == 'Diff':
            cin = av * H.sum(v - x[0][H.tgt]) + bv
        elif cfname == 'Sigmoidal':
            q = {k: _f32(cf.param[k]) for k in ('cmax', 'midpoint', 'r')}
            cin = av * H.sum(q['cmax'] / (1 + torch.exp(q['r'] * (q['midpoint'] - v))))
        else:
            cin = av * H.sum(v) + bv
        f = _drift(name, x, cin, p, m)
        new = [x[k] + dt * f[k] for k in range(ns)]
        if noise:
            new = [new[k] + sq * sig[k] * z[(t % spc) * ns + k] for k in range(ns)]
        if name == 'Kuramoto':
            new[0] = _wrap(new[0])
        elif name == 'MPR':
            new[0] = torch.clamp(new[0], min=0.0)
        if bold:
            bst = _balloon(bst, torch.sin(x[0]) if name == 'Kuramoto' else x[0], _f32(DT / 1000.0))
            if (t + 1) % bold == 0:
                rows.append(_bold_signal(bst[2], bst[3]).T)
        live = t < last
        x = [torch.where(live, new[k], x[k]) for k in range(ns)]
    state = torch.stack(x).permute(2, 1, 0).contiguous()
    return state, (torch.stack(rows, 1) if rows else None)


def _fc_exact(x, target):
    c = x - x.mean(1, keepdim=True)
    g = c.transpose(1, 2) @ c
    s = torch.sqrt(torch.diagonal(g, dim1=1, dim2=2))
    fc = g / (s[:, :, None] * s[:, None, :])
    iu = torch.triu_indices(fc.shape[1], fc.shape[1], 1, device='cuda')
    return [fc, ((fc - target)[:, iu[0], iu[1]] ** 2).sum(1)]


def _exact_step(c, seed):
    conn, lnz, ntime, th, par, obs, a = _step_inputs(c, seed)
    one = c['subjects'] == 1
    x = torch.from_numpy(th[None] if one else th).cuda().to(F64)[:, :, 0]
    om = torch.from_numpy(par[None] if one else par).cuda().to(F64)[:, :, 0]
    ob = torch.from_numpy(obs[:, None] if one else obs).cuda().to(F64)
    av = torch.as_tensor(np.atleast_1d(np.asarray(a, np.float32)), device='cuda').to(F64)[:, None]
    row = np.asarray(conn.row, np.int64)
    tgt = torch.from_numpy(np.repeat(np.arange(c['N']), np.diff(row))).cuda()
    col = torch.from_numpy(np.asarray(conn.col, np.int64)).cuda()
    d = torch.from_numpy(lnz.astype(np.int64)).cuda()
    w = torch.from_numpy(np.asarray(conn.wnz, np.float32)).cuda().to(F64)
    for k in range(c['nstep']):
        t = ntime + k
        # the network reads row t before the model writes it
        s = torch.sin(ob[torch.remainder(t - d, ntime), :, col, 0].T - ob[t % ntime, :, :, 0][:, tgt])
        cin = torch.zeros_like(x).index_add_(1, tgt, s * w) / c['N'] * av
        ob[t % ntime, :, :, 0] = x
        ob[t % ntime, :, :, 1] = torch.sin(x)
        x = _wrap(x + om + cin)
    x = x[:, :, None]
    return [x[0] if one else x, ob[:, 0] if one else ob]


def _exact_lems(c, seed):
    conn, params, x0 = _lems_inputs(c, seed)
    I, N, ns = x0.shape
    dt = np.float32(DT)
    rec = (np.float32(1.0) / params[:, 0]).astype(np.float32) / dt
    uniq, tab = np.unique(rec, return_inverse=True)
    D = np.stack([(np.asarray(conn.lnz, np.float32) * r).astype(np.int64) for r in uniq], 1)
    H = _History(conn, D[:, tab], N, I)
    g = torch.from_numpy(params[:, 1]).cuda().to(F64)[None, :]
    x = list(torch.from_numpy(x0).cuda().to(F64).permute(2, 1, 0).contiguous())
    amp = _f32(dt) ** 0.5 * 2e-6 ** 0.5
    lim = [(-2, 1), (-20, 2), (-2, 5), (-2, 0), (0, 2), (-1, 1)]
    inst = torch.arange(I, device='cuda')
    for t in range(c['nsteps']):
        z = torch.cat([_normals(N, inst, t, seed, b) for b in (0, 1)])
        x1, y1, zz, x2, y2, gg = x
        H.write(t, x1)
        cpop = g * H.sum(torch.sin(H.read(t) - x1[H.tgt]))
        fx1 = torch.where(x1 < 0, -x1 * x1 + 3 * x1, -x2 + 0.6 * (zz - 4) ** 2)
        hz = 4 * (x1 + 1.6) + torch.where(zz < 0, -0.1 * zz ** 7, torch.zeros_like(zz))
        fy2 = torch.where(x2 < -0.25, torch.zeros_like(x2), 6 * (x2 + 0.25))
        f = [y1 - zz + 3.1 + 0.1 * cpop + fx1 * x1, 1 - 5 * x1 * x1 - y1,
             0.00035 * (hz - zz - 0.2 * cpop),
             -y2 + x2 - x2 ** 3 + 0.45 + 2 * gg - 0.3 * (zz - 3.5), (-y2 + fy2) / 10,
             -0.01 * (gg - 0.1 * x1)]
        x = [torch.clamp(x[k] + _f32(dt) * f[k] + amp * z[k], *lim[k]) for k in range(ns)]
    state = torch.stack(x).permute(2, 1, 0).contiguous()
    return [state, (state[:, :, 3] - state[:, :, 0])[:, :, None]]


def _exact_net(c, seed):
    conn, x0 = _net_inputs(c, seed)
    m, _ = _make('Generic2dOscillator', 'Linear')
    d = network.delays_f32(conn.lnz, 4.0, DT, 'ceil')
    H = _History(conn, d, c['N'], 1)
    x = list(torch.from_numpy(x0).cuda().to(F64).T.contiguous()[:, :, None])
    p = [_f32(m.const['a'])]
    for t in range(c['nsteps']):
        H.write(t, x[0])
        f = _drift('Generic2dOscillator', x, _f32(0.05) * H.sum(H.read(t)), p, m)
        x = [x[k] + _f32(DT) * f[k] for k in range(2)]
    return [torch.stack(x)[:, :, 0].T.contiguous()]


def _exact_fit(c, seed):
    conn, x0, eta, G, target = _fit_inputs(c, seed)
    I, N, T = c['I'], c['N'], c['T']
    m = model.MPR()
    k = {n: _f32(v) for n, v in m.const.items()}
    dt, tau = _f32(DT), k['tau']
    H = _History(conn, network.delays_f32(conn.lnz, 4.0, DT, 'ceil'), N, I)
    r, V = torch.from_numpy(x0).cuda().to(F64).permute(2, 1, 0).contiguous()
    et = torch.from_numpy(eta).cuda().to(F64).T
    Gv = torch.from_numpy(G).cuda().to(F64)[None, :]
    R, Vs, Ss, clamped = [r], [V], [], []
    for t in range(T):
        H.write(t, r)
        S = H.sum(H.read(t))
        fr, fV = _drift('MPR', [r, V], Gv * S, [et], m)
        rn = r + dt * fr
        clamped.append(rn < 0)
        r, V = torch.clamp(rn, min=0.0), V + dt * fV
        R.append(r)
        Vs.append(V)
        Ss.append(S)
    X = torch.stack(R[1:]).permute(2, 0, 1).contiguous().requires_grad_()
    fc = _fc_exact(X, 0.0)[0]
    tg = torch.from_numpy(target).cuda().to(F64)
    iu = torch.triu_indices(N, N, 1, device='cuda')
    loss = ((fc - tg)[:, iu[0], iu[1]] ** 2).mean(1)
    dr = torch.autograd.grad(loss.sum(), X)[0].permute(1, 2, 0)      # [T, N, I]
    loss = loss.detach()
    mu = torch.zeros((T + 2 + int(H.d.max()), N, I), dtype=F64, device='cuda')
    lr, lv = dr[T - 1].clone(), torch.zeros((N, I), dtype=F64, device='cuda')
    deta = torch.zeros((N, I), dtype=F64, device='cuda')
    dG = torch.zeros((N, I), dtype=F64, device='cuda')
    for t in range(T - 1, -1, -1):
        mr, mv = torch.where(clamped[t], torch.zeros_like(lr), lr), lv
        mu[t + 1] = mv
        v = mu.view(-1, I)[(t + 1 + H.d) * N + H.tgt]
        coup = torch.zeros((N, I), dtype=F64, device='cuda').index_add_(0, H.col, H.w * v)
        rr, VV = R[t], Vs[t]
        deta += dt / tau * mv
        dG += dt / tau * mv * Ss[t]
        lr = (mr + dt * (mr * 2 * VV / tau + mv * (k['J'] * tau - 2 * (math.pi * tau) ** 2 * rr) / tau)
              + dt * Gv / tau * coup + (dr[t - 1] if t > 0 else 0.0))
        lv = mv + dt * (mr * 2 * rr / tau + mv * 2 * VV / tau)
    return [loss, dG.sum(0), deta.T.contiguous()]


def exact(case, seed):
    c = case
    kind = c['kind']
    if kind == 'step':
        return _exact_step(c, seed)
    if kind in ('sweep', 'instances'):
        conn, x0, par, a, sp, target = _sweep_inputs(c, seed)
        bold = c.get('bold', 0)
        state, rows = _simulate(c['model'], c['cfun'], conn, x0, par, a, sp, c['nsteps'], c['noise'],
                                seed, bold)
        if not bold:
            return [state]
        return [state, rows] + _fc_exact(rows, torch.from_numpy(target).cuda().to(F64))
    if kind == 'batch':
        return [_simulate('MPR', 'Linear', conn, x0, eta, a, np.full(a.size, 4.0, np.float32), steps,
                          True, sd)[0] for conn, x0, eta, a, steps, sd in _batch_parts(c, seed)]
    if kind == 'lems':
        return _exact_lems(c, seed)
    if kind == 'net':
        return _exact_net(c, seed)
    if kind == 'adjoint':
        return _exact_fit(c, seed)
    if kind == 'fc':
        x = _series(c['I'], c['T'], c['N'], seed).to(F64)
        return _fc_exact(x, torch.from_numpy(_target(c['N'], seed)).cuda().to(F64))
    if kind == 'stream':
        x = _series(c['I'], c['rows'], c['N'], seed).to(F64)
        u = x - x.mean(1, keepdim=True)
        m2 = u.transpose(1, 2) @ u
        if c['rows'] < 2:
            return [x.mean(1), m2, None]    # one sample has no correlation
        s = torch.sqrt(torch.diagonal(m2, dim1=1, dim2=2))
        return [x.mean(1), m2, m2 / (s[:, :, None] * s[:, None, :])]
    rmap, node = _rmap_inputs(c, seed)
    roi = torch.zeros((c['nroi'], c['nvar']), dtype=F64, device='cuda').index_add_(
        0, rmap.long(), node.to(F64))
    return [roi, roi[rmap.long()]]
