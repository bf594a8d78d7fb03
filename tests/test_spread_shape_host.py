"""
The default launch shape of a group set (groups.spread_shape) over what the
device reports as resident clusters, without a device: a shape of which no
cluster can be resident is never taken, and the plain kernel is where none can.
"""

import types

import numpy as np
import pytest

from tvb_hpc import autotune, groups, _native as nat

SMS = 152


def shape(monkeypatch, N, G, resident, channels=1, cfun=nat.CFUN_LINEAR):
    "spread_shape of G groups where resident(threads, cluster) clusters fit the device."
    monkeypatch.setattr(autotune, 'group_max_clusters', lambda s, t, c, tpn=1, n=0: resident(t, c))
    s = types.SimpleNamespace(cfun_id=cfun, N=N, n_groups=G, can_pipeline=True, pipelined_built=True, channels=channels,
                              pipe_tab=np.array([True]), gtab=np.zeros(G, int))
    return groups.spread_shape(s, SMS)


@pytest.mark.parametrize('channels', [1, 2])
@pytest.mark.parametrize('N', [16, 68, 84, 192, 400, 512, 998])
@pytest.mark.parametrize('G', [1, 10, 100, 400])
@pytest.mark.parametrize('largest', [0, 1, 2, 4, 8, 16])
def test_only_shapes_that_fit(monkeypatch, N, G, channels, largest):
    got = shape(monkeypatch, N, G, lambda t, c: SMS // c if c <= largest else 0, channels)
    plain = groups.plain_shape(N, G, SMS) + (0, 1)
    assert got == plain or (got[3] == groups.PIPELINED and got[1] <= largest)
    if largest == 0:
        assert got == plain


def test_choice_where_every_cluster_fits(monkeypatch):
    "The measured choices: few groups spread out, many on the smallest cluster of the wider build."
    free = lambda t, c: SMS // c
    assert shape(monkeypatch, 84, 32, free) == (384, 4, 0, groups.PIPELINED)
    assert shape(monkeypatch, 84, 400, free)[:2] == (704, 2)
    assert shape(monkeypatch, 192, 400, free)[:2] == (768, 4)
    assert shape(monkeypatch, 998, 400, free)[:2] == (1024, 16)


@pytest.mark.parametrize('N', [30, 84, 200, 400, 700])
def test_sigmoidal_sets_beyond_residency_are_plain(monkeypatch, N):
    """The Sigmoidal gather is bound by its exponentials: pipelined only where every
    group's cluster is resident at once on an SM each."""
    for G in (1, 8, 64, 512):
        got = shape(monkeypatch, N, G, lambda t, c: SMS // c, cfun=nat.CFUN_SIGMOIDAL)
        if got[3] == groups.PIPELINED:
            assert G * got[1] <= SMS
        else:
            assert got == groups.plain_shape(N, G, SMS) + (0, 1)
    assert shape(monkeypatch, N, 1, lambda t, c: SMS // c, cfun=nat.CFUN_SIGMOIDAL)[3] == groups.PIPELINED
