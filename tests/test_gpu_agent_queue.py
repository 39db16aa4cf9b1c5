"""The agent pass with the efficacy queue (large states) and without, against the standalone
check_immunity on the same state: the same arrays, records and sums."""
import numpy as np
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L

pytestmark = pytest.mark.gpu


# in place, and above the queue's threshold (12 agent blocks of 256 a resident block, four blocks an SM)
@pytest.mark.parametrize('n', [8_021, 1_950_011])
def test_agent_pass_efficacies_equal_check_immunity(n):
    day = 24
    sim = cv.Sim(dict(pop_size=n, pop_type='random', n_days=40, pop_infected=n // 8, rand_seed=3, n_variants=1),
                 gpu_population=True)
    sim.initialize()
    sim._seed()
    st = sim.state
    st.run_days(0, day, close_last=False, use_graph=False)
    st.agent_step(day, True, True, steady=True)
    got = {k: st.t[k].clone() for k in ('sus_imm', 'symp_imm', 'sev_imm')}
    rec = st.t['tgt_rec'].clone()
    assert (got['sus_imm'] > 0).float().mean() > 0.02
    st.check_immunity(day)
    for k, x in got.items():
        assert torch.equal(x, st.t[k]), k
    sus = st.get('susceptible')
    want = st.t['rel_sus'] * (1 - got['sus_imm'][0])
    assert torch.equal(rec[0][:n][sus].abs(), want[:n][sus])
    fx = st.res_fx.view(sim.npts, L.N_RES_F)[day].cpu().numpy()
    for col, k in ((1, 'sus_imm'), (2, 'symp_imm')):
        assert fx[col] == int(torch.round(got[k].double() * 2.0 ** L.FX_IMM_BITS).long().sum())
    assert st.status() == 0 and np.isfinite(fx).all()
