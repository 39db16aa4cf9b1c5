"""The autotuner times the stored layers' pass, so what decides whether and beside what that pass
runs is part of the key its choice is kept under, and a state that never runs it is not timed."""
from types import SimpleNamespace

import pytest

from covasim_gb300 import _lib as L
from covasim_gb300 import autotune


def make_state(src_walk=0, has_testing=False, lik_active=False, label='2048w'):
    segments = [SimpleNamespace(n_edges=1000, dynamic=0), SimpleNamespace(n_edges=500, dynamic=1)]
    return SimpleNamespace(segments=segments, n=500, specs=[SimpleNamespace(npts=10)], device='cuda:0',
                           cstate=SimpleNamespace(src_walk=src_walk), has_testing=has_testing, lik_active=lik_active,
                           edge_tile_label=label, snapshot=lambda: {}, set_edge_tile=lambda **k: None, restore=lambda s: None)


@pytest.fixture(autouse=True)
def device(monkeypatch):
    monkeypatch.setattr(autotune.torch.cuda, 'get_device_name', lambda d: 'a GPU')
    monkeypatch.setattr(autotune, '_CACHE', {})


@pytest.mark.parametrize('other', [dict(src_walk=32), dict(src_walk=-1), dict(has_testing=True), dict(lik_active=True)])
def test_states_that_run_the_pass_differently_have_their_own_key(other):
    assert autotune.workload_signature(make_state(**other)) != autotune.workload_signature(make_state())
    assert autotune.workload_signature(make_state(**other)) == autotune.workload_signature(make_state(**other))


def test_a_state_that_walks_every_layer_is_not_timed(monkeypatch, tmp_path):
    monkeypatch.setattr(autotune, '_candidates', lambda *a: pytest.fail('candidates of a pass that does not run'))
    cache = tmp_path / 'tuned.json'
    best, ms = autotune.tune_edge_tile(make_state(src_walk=L.WALK_ALL, label=4096), cache_file=str(cache))
    assert (best, ms) == ('4096', {}) and not autotune._CACHE and not cache.exists()
