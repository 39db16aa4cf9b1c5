"""The test pass that marks the traced agents' contacts itself against the same marks made
by the passes of their own (as a tracing capacity needs them)."""
import numpy as np
import pytest
import torch

import covasim_gb300 as cv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('pop_type,n,dyn,presumptive', [('random', 33, False, False), ('random', 257, True, True),
                                                        ('hybrid', 2049, True, False), ('hybrid', 20_001, False, True)])
def test_marks_in_the_test_pass_equal_the_separate_passes(pop_type, n, dyn, presumptive):
    runs = []
    for separate in (False, True):
        pars = dict(pop_type=pop_type, pop_size=n, n_days=40, rand_seed=5, pop_infected=min(20, n // 3),
                    interventions=[cv.test_prob(symp_prob=0.5, asymp_prob=0.05),
                                   cv.contact_tracing(trace_probs=0.8, trace_time=1, presumptive=presumptive)])
        if dyn:
            pars['dynam_layer'] = dict(h=0, s=0, w=0, c=1) if pop_type == 'hybrid' else dict(a=1)
        sim = cv.Sim(pars)
        sim.initialize()
        assert sim.state.cstate.has_testing == 1 | 8 | 16
        if separate:  # the capacity bit without a capacity in any sim; the day's preparation runs too
            sim.state.cstate.has_testing = 1 | 4 | 8
        sim.run(use_graph=False)
        st = sim.state
        runs.append((sim.raw_results(), [st.t[k].clone() for k in ('flags', 'dates', 'pending_quar', 'contact_bits')]))
    for key in runs[0][0]:
        np.testing.assert_array_equal(runs[0][0][key], runs[1][0][key], err_msg=key)
    assert all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(runs[0][1], runs[1][1]))
    assert runs[0][0]['new_quarantined'].sum() > 0 or n < 300
