"""A tracing capacity on the days after test_prob's last one, when the diagnoses it left behind
(test_delay) are still being traced: the day's cases alone count against it."""
import pytest

import covasim_gb300 as cv
from oracle.interventions import TestProb, ContactTracing
from test_gpu_sim import compare_runs, oracle_for
from test_gpu_testing import TESTING_KEYS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dyn', [False, True])
def test_capacity_after_testing_has_ended(dyn):
    tp = dict(symp_prob=0.5, asymp_prob=0.05, test_delay=5, end_day=25)
    ct = dict(trace_probs=0.8, trace_time=1, capacity=5)
    pars = dict(pop_type='hybrid', pop_size=3000, n_days=45, rand_seed=12, pop_infected=300)
    if dyn:
        pars['dynam_layer'] = dict(h=0, s=0, w=0, c=1)
    sim = cv.Sim(dict(pars, interventions=[cv.test_prob(**tp), cv.contact_tracing(**ct)]))
    sim.initialize()
    orc = oracle_for(sim)
    orc.interventions = [TestProb(**tp), ContactTracing(**ct)]
    for iv in orc.interventions:
        if hasattr(iv, 'initialize'):
            iv.initialize(orc)
    orc.run()
    sim.run()
    for day in range(26, 31):  # more cases than the capacity, on days without tests
        assert (orc.people.date_diagnosed == day).sum() > 5
    compare_runs(sim, orc, keys=TESTING_KEYS)
