"""
tvbg_rmap_to_avg at the edges of its parts: groups of 32 nodes, parts per
warp and CTA, bins per cluster (1600) and variables per cluster (32); sorted,
random and one-region maps with entries outside [0, nroi).

Tolerance: a sum passes at most 5 (tree) + 32 (turns of a group) + 40 (groups
of a warp) float32 additions: 77 * 2^-24 < 6e-6 of the sum of |x|.
"""

import numpy as np
import pytest

from tvb_hpc import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind', ['sorted', 'random', 'one'])
@pytest.mark.parametrize('nnode,nroi,nvar', [(1, 1, 1), (31, 3, 2), (33, 5, 1), (4096, 1600, 1),
                                             (4097, 1601, 1), (5000, 70, 33), (40001, 3, 70),
                                             (20000, 5000, 3), (131073, 68, 2)])
def test_to_avg(cuda, kind, nnode, nroi, nvar):
    torch = cuda
    rng = np.random.default_rng(nnode + nroi)
    rmap = rng.integers(-1, nroi + 1, nnode).astype(np.int32)
    if kind == 'sorted':
        rmap.sort()
    elif kind == 'one':
        rmap[:] = nroi - 1
    node = rng.normal(size=(nnode, nvar)).astype(np.float32)
    roi = torch.full((nroi, nvar), float('nan'), device='cuda')
    args = dict(nroi=nroi, nvar=nvar, nnode=nnode, rmap=torch.from_numpy(rmap).cuda(),
                node=torch.from_numpy(node).cuda())
    network.RMapToAvg().kernel()(roi=roi, **args)
    ref, mag = np.zeros((nroi, nvar)), np.zeros((nroi, nvar))
    ok = (rmap >= 0) & (rmap < nroi)
    np.add.at(ref, rmap[ok], node[ok].astype(np.float64))
    np.add.at(mag, rmap[ok], np.abs(node[ok]).astype(np.float64))
    got = roi.cpu().numpy()
    assert np.all(np.abs(got - ref) <= 6e-6 * mag)
    again = torch.empty_like(roi)
    network.RMapToAvg().kernel()(roi=again, **args)
    assert np.array_equal(again.cpu().numpy(), got)
