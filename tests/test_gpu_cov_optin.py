"""
Streaming-FC updates whose shared memory lies next to the 48 KB that a launch
takes without opting in (dynamic 8 N (1 + 2 rows) bytes and the static tile of
8448), as the first calls of a process: an earlier, larger update leaves the
kernel's limit raised.

Tolerance: FP64 sums of at most 16 products, 16 * 2^-52 < 1e-14 of the sum of
magnitudes, 1e-13 here; the means take one rounding per sample (1e-14).
"""

import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

# (nodes, rows): dynamic bytes 40704 (the last that needs no opt-in) to 49152
SIZES = [(1696, 1), (1697, 1), (1800, 1), (2048, 1), (566, 4), (330, 8), (300, 8), (361, 8), (270, 10),
         (220, 12), (245, 12), (170, 16)]


def dynamic_bytes(N, rows):
    return 8 * N * (1 + 2 * rows)


def test_sizes_lie_at_the_limit():
    assert dynamic_bytes(*SIZES[0]) + 8448 == 48 * 1024
    assert all(48 * 1024 < dynamic_bytes(N, r) + 8448 and dynamic_bytes(N, r) <= 48 * 1024
               for N, r in SIZES[1:])


def first_calls():
    import torch
    from tvb_hpc import metric
    bad = []
    for N, rows in SIZES:
        try:
            x = (1.0 + 0.1 * np.random.default_rng(N).normal(size=(2, 2 * rows, N))).astype(np.float32)
            xd = torch.from_numpy(x).cuda()
            fc = metric.StreamingFC(2, N)
            for r in range(0, 2 * rows, rows):
                if rows == 1:
                    fc.update(xd[:, r])
                else:
                    fc.update_rows(xd, range(r, r + rows))
            x = x.astype(np.float64)
            u = x - x.mean(axis=1, keepdims=True)
            ref = np.einsum('bti,btj->bij', u, u)
            mag = np.sqrt(np.einsum('bii->bi', ref))
            assert np.all(np.abs(fc.m2.cpu().numpy() - ref) <= 1e-13 * mag[:, :, None] * mag[:, None, :] * 2 * rows)
            np.testing.assert_allclose(fc.mean.cpu().numpy(), x.mean(axis=1), rtol=1e-14)
        except Exception as e:
            bad.append((N, rows, repr(e)[:200]))
    assert not bad, bad


@pytest.mark.gpu
def test_first_calls(cuda):
    code = ('import sys; sys.path[:0] = [%r, %r]; import test_gpu_cov_optin as t; t.first_calls()'
            % (os.path.join(ROOT, 'tests'), os.path.join(ROOT, 'tvb-hpc_gb300')))
    p = subprocess.run([sys.executable, '-c', code], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-3000:]
