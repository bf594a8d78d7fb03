"""
Region sums of few nodes, where a CTA per region scans the map, and on both
sides of the line to the cluster kernel; against FP64.

Tolerance: the scan adds in pairs of float32 words and rounds once (2^-24, 1.2e-7 with a
margin of two); the cluster as in test_gpu_rmap_edges.py (6e-6).
"""

import numpy as np
import pytest

from tvb_hpc import network

pytestmark = pytest.mark.gpu


# scan: whether the call lies on the scan's side of the line
@pytest.mark.parametrize('nnode,nroi,nvar,scan', [
    (1, 1, 1, True), (255, 3, 5, True), (257, 68, 4, True), (4000, 400, 6, True), (5000, 9000, 1, True),
    (100, 3, 700, True), (8800, 2, 1, True), (9100, 2, 1, False), (30000, 1600, 1, True), (5000, 20000, 1, False),
    (70001, 1600, 1, False), (70001, 1601, 1, False), (70001, 70, 33, False), (100, 3, 70000, False)])
def test_region_sums(cuda, nnode, nroi, nvar, scan):
    torch = cuda
    rng = np.random.default_rng(nnode + nroi)
    rmap = rng.integers(-1, nroi + 1, nnode).astype(np.int32)
    node = rng.normal(size=(nnode, nvar)).astype(np.float32)
    roi = torch.full((nroi, nvar), float('nan'), device='cuda')
    network.RMapToAvg().kernel()(nroi=nroi, nvar=nvar, nnode=nnode, rmap=torch.from_numpy(rmap).cuda(),
                                 node=torch.from_numpy(node).cuda(), roi=roi)
    ref, mag = np.zeros((nroi, nvar)), np.zeros((nroi, nvar))
    ok = (rmap >= 0) & (rmap < nroi)
    np.add.at(ref, rmap[ok], node[ok].astype(np.float64))
    np.add.at(mag, rmap[ok], np.abs(node[ok]).astype(np.float64))
    tol = 1.2e-7 if scan else 6e-6
    assert np.all(np.abs(roi.cpu().numpy() - ref) <= tol * mag)
