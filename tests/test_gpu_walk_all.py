"""The default rule that walks every stored layer on every day (no tile pass) against the
streamed pass, at sizes around the per-source passes' warp splits."""
import numpy as np
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('pop_type,n,dyn,trace', [('random', 31, True, False), ('hybrid', 1000, True, False),
                                                  ('hybrid', 66_001, True, False), ('hybrid', 20_001, False, True),
                                                  ('random', 530_003, False, True)])
def test_walk_every_day_equals_streamed(pop_type, n, dyn, trace):
    """Busy and quiet days; a redrawn layer beside the stored ones, or tracing through the index."""
    runs = []
    for mode in (None, 0):
        pars = dict(pop_type=pop_type, pop_size=n, n_days=30 if n > 100_000 else 60, rand_seed=8,
                    pop_infected=max(5, n // 50), n_imports=2, interventions=[])
        if dyn:
            pars['dynam_layer'] = dict(h=0, s=0, w=0, c=1) if pop_type == 'hybrid' else dict(a=1)
        if trace:
            pars['interventions'] = [cv.test_prob(symp_prob=0.3), cv.contact_tracing(trace_probs=0.5)]
        sim = cv.Sim(pars)
        sim.initialize()
        if mode is None:
            assert sim.state.cstate.src_walk == (32 if dyn else (L.WALK_ALL if n >= 150_000 else 0))
            sim.state.set_src_walk(-1)
            assert sim.state.cstate.src_walk == L.WALK_ALL
        else:
            sim.state.set_src_walk(mode)
        sim.run(use_graph=False)
        runs.append((sim.raw_results(), [sim.state.t[k].clone() for k in ('flags', 'vstate', 'dates')],
                     sim.state.infection_log_tensor(0)))
    for key in runs[0][0]:
        np.testing.assert_array_equal(runs[0][0][key], runs[1][0][key], err_msg=key)
    assert all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(runs[0][1], runs[1][1]))
    assert torch.equal(runs[0][2], runs[1][2])
    assert runs[0][0]['new_infections'].sum() > 0 or n < 100


def test_walk_takes_weighted_edges_and_several_layers():
    rng = np.random.default_rng(0)
    n = 3000
    layers = {}
    for key, m in (('a', 9000), ('b', 4001), ('c', 1)):
        p1, p2 = np.sort(rng.integers(0, n, m)), rng.integers(0, n, m)
        layers[key] = dict(p1=p1.astype(np.int32), p2=p2.astype(np.int32), beta=rng.random(m).astype(np.float32))
    popdict = dict(uid=np.arange(n), age=rng.integers(0, 90, n).astype(float), sex=rng.integers(0, 2, n),
                   contacts=layers)
    out = []
    for mode in (-1, 0):
        sim = cv.Sim(dict(pop_size=n, n_days=40, pop_infected=40, rand_seed=2, beta=0.2, contacts=dict(a=1, b=1, c=1),
                          beta_layer=dict(a=1.0, b=0.5, c=2.0), iso_factor=dict(a=1, b=1, c=1),
                          quar_factor=dict(a=1, b=1, c=1), dynam_layer=dict(a=0, b=0, c=0)),
                     popdict={**popdict, 'contacts': {k: dict(v) for k, v in layers.items()}})
        sim.initialize()
        sim.state.set_src_walk(mode)
        assert sim.state.cstate.src_walk == (L.WALK_ALL if mode else 0)
        sim.run(use_graph=False)
        out.append(sim.raw_results())
    for key in out[0]:
        np.testing.assert_array_equal(out[0][key], out[1][key], err_msg=key)
    assert out[0]['new_infections'].sum() > 500
