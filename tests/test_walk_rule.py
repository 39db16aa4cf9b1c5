"""The default walk rule (BatchState._walk_mode): by the day's prevalence in large states, with
testing as without, since testing need not keep an epidemic small; every day in the others."""
from types import SimpleNamespace

import pytest

from covasim_gb300 import _lib as L
from covasim_gb300.state import BatchState


def mode(n, dynamic, testing, edges_per_agent=17.75, sims=1, src_walk=0, asked=False, lik=False, indexed=True):
    segments = [SimpleNamespace(dynamic=0, rp1=1 if indexed else None, n_edges=int(n * edges_per_agent))]
    if dynamic:
        segments.append(SimpleNamespace(dynamic=1, rp1=None, n_edges=10 * n))
    state = SimpleNamespace(src_walk=128 if dynamic and not asked else src_walk, segments=segments, n=n, specs=[None] * sims,
                            has_testing=testing, lik_active=lik, _walk_default=not asked)
    return BatchState._walk_mode(state)


@pytest.mark.parametrize('sims', [1, 16])
@pytest.mark.parametrize('n', [350_000, 420_000, 1_000_000, 10_000_000])
def test_large_states_with_a_redrawn_layer_go_by_prevalence(n, sims):
    assert 16 <= mode(n, True, True, sims=sims) <= 128
    assert 16 <= mode(n, True, False, sims=sims) <= 128


@pytest.mark.parametrize('n', [20_000, 349_999])
def test_small_states_with_a_redrawn_layer(n):
    assert mode(n, True, True) == mode(n, True, True, sims=16) == L.WALK_ALL  # one launch a day instead of two
    assert mode(n, True, False) == mode(n, True, False, sims=16) == 32


@pytest.mark.parametrize('n,edges,want', [(20_000, 17.75, 0), (399_999, 17.75, 0), (400_000, 17.75, 32), (899_999, 17.75, 32),
                                          (900_000, 17.75, L.WALK_ALL), (4_000_000, 17.75, L.WALK_ALL), (149_999, 10, 0),
                                          (150_000, 10, L.WALK_ALL), (500_000, 12.5, 32)])
def test_testing_without_a_redrawn_layer(n, edges, want):
    assert mode(n, False, True, edges) == want


def test_what_was_asked_for_and_the_likelihood():
    assert mode(1_000_000, True, True, asked=True, src_walk=-1) == L.WALK_ALL
    assert mode(1_000_000, True, True, asked=True, src_walk=-1, indexed=False) == -1
    assert mode(1_000_000, True, True, asked=True, src_walk=8) == 8
    assert mode(1_000_000, True, True, lik=True) == 128
    assert mode(2_000_000, False, False, sims=24, src_walk=64) == L.WALK_ALL
    assert mode(2_000_000, False, False, sims=24) == 0
