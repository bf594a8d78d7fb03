"""
Residency that tvbg_group_occupancy and tvbg_group_max_clusters report, against
the registers of the builds that launches take: pipelined CTAs of at most 512
threads have a build of up to 128 registers a thread and one of at most 80, and
a launch takes the second where it needs fewer waves of CTAs.
"""

import ctypes

import numpy as np
import pytest

from tvb_hpc import autotune, groups, model, coupling, network, scheme, _native as nat

pytestmark = pytest.mark.gpu


def group_set():
    w, ln = network.synthetic_connectome(16, 0.5, seed=0)
    m = model.MPR()
    return groups.GroupSet(m, coupling.Linear(m), scheme.EulerStep(0.1), network.Connectivity.from_dense(w, ln),
                           dt=0.1, couplings=np.full(8, 0.1), speeds=1.0,
                           state0=np.zeros((8, 16, 2), np.float32))


@pytest.mark.parametrize('threads', [128, 192, 256, 320, 384, 512])
def test_pipelined_residency(cuda, threads):
    s = group_set()
    s.set_shape(256, 1, 0, 2)
    cfg = s.launch_cfg(8)
    cfg.threads = threads
    per, sms = groups.group_occupancy(cfg)
    wide, mid = 512 // threads, 65536 // (80 * threads)      # CTAs an SM's registers hold
    assert sms == groups.device_sms()
    assert per == max(wide, mid)
    # clusters of one CTA: a launch that the wide build holds at once, and one that it does not
    assert autotune.group_max_clusters(s, threads, 1, 2) == per * sms
    assert autotune.group_max_clusters(s, threads, 1, 2, wide * sms) == wide * sms
    assert autotune.group_max_clusters(s, threads, 1, 2, wide * sms + 1) == per * sms
    n = ctypes.c_int32()
    cfg.tpn, cfg.cluster = 2, 1
    nat.check(nat.load().tvbg_group_max_clusters(ctypes.byref(cfg), ctypes.byref(n)))
    assert n.value == per * sms
    assert nat.load().tvbg_group_max_clusters_for(ctypes.byref(cfg), -1, ctypes.byref(n)) == nat.TVBG_EINVAL
