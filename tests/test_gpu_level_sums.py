"""The fixed-point sums of the agents' levels, over every level that a state can be given."""
import numpy as np
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('levels', [[0.0, 1.5, -1.5], [127.9, 128.0, 128.1, 5000.25], [-127.9, -128.0, -128.1, -5000.25]])
def test_nab_sum_is_the_sum_of_the_rounded_levels(levels):
    n = 3001
    sim = cv.Sim(dict(pop_size=n, pop_type='random', n_days=5, pop_infected=0, rand_seed=1))
    sim.initialize()
    st = sim.state
    nab = np.resize(np.asarray(levels, np.float32), n)
    st.set('nab', nab)  # no peak: the levels stay as they are
    st.agent_step(1, True, True)
    want = np.rint(nab.astype(np.float64) * 2.0 ** L.FX_NAB_BITS).astype(np.int64).sum()
    assert int(st.res_fx.view(sim.npts, L.N_RES_F)[0, 0].item()) == want
    assert torch.equal(st.get('nab').cpu(), torch.from_numpy(nab))
