"""The agent pass with the efficacy queue over a batch of uneven sims (the queue is emptied where a
warp's agent blocks change sims), with several variants and vaccinated agents, and in place."""
import numpy as np
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L
from covasim_gb300.state import ff_log

pytestmark = pytest.mark.gpu
DAY = 24


def _vaccinate(st, gen):
    """A third of every sim's agents vaccinated, two products with efficacies of their own."""
    keep = []
    for k, (r, sp) in enumerate(zip(st.sim_recs, st.specs)):
        vx = (0.1 + 0.9 * torch.rand((2, sp.nv), generator=gen)).to(torch.float32)
        ln = torch.tensor([ff_log(float(x)) for x in vx.flatten()], dtype=torch.float32)
        keep += [vx.cuda(), ln.cuda()]
        r.vx_imm, r.vx_ln_imm, r.n_vaccines = keep[-2].data_ptr(), keep[-1].data_ptr(), 2
        on = torch.rand(sp.n, generator=gen) < 1 / 3
        st.set('vaccinated', on.numpy(), sim=k)
        st.set('vaccine_source', torch.randint(0, 2, (sp.n,), generator=gen).numpy(), sim=k)
        have = st.get('nab', k).cpu()
        level = torch.where(on, have + 3 * torch.rand(sp.n, generator=gen), have)
        st.set('nab', level.numpy(), sim=k)
        st.set('peak_nab', torch.where(on, level, st.get('peak_nab', k).cpu()).numpy(), sim=k)
    recs = (L.SimParams * len(st.sim_recs))(*st.sim_recs)
    st.sims_dev.copy_(torch.frombuffer(bytearray(bytes(recs)), dtype=torch.uint8))
    return keep


# in place; and past the queue's line of 12 agent blocks of 256 a resident block, four of those an SM
@pytest.mark.parametrize('sizes', [(31, 8_021, 257, 4_000), (33, 700_001, 1, 1_000, 611_003, 255, 599_999, 31, 8_021)])
def test_uneven_sims_variants_and_vaccinated(sizes):
    sims = [cv.Sim(dict(pop_size=n, pop_type='random', n_days=40, pop_infected=max(1, n // 8), rand_seed=k),
                   gpu_population=True,
                   variants=[cv.variant('b117', days=0, n_imports=0), cv.variant('p1', days=0, n_imports=0)] if k % 3 else [])
            for k, n in enumerate(sizes)]
    b = cv.BatchSim(sims).initialize()
    b.seed_infections()
    st = b.state
    line = 12 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    assert (st.n_agent_blocks >= line) == (sum(sizes) > 10**6)
    st.run_days(0, DAY, close_last=False, use_graph=False)
    gen = torch.Generator().manual_seed(1)
    for k, sp in enumerate(st.specs):  # the recovered had any of the variants
        rv = st.get('recovered_variant', k).cpu().numpy()
        st.set('recovered_variant', np.where(np.isnan(rv), rv, np.arange(sp.n) % sp.nv), sim=k)
    keep = _vaccinate(st, gen)
    fx0 = st.res_fx.clone()
    st.agent_step(DAY, True, True)
    keys = ('sus_imm', 'symp_imm', 'sev_imm')
    got = {key: [st.get(key, k).clone() for k in range(len(sizes))] for key in keys}
    rec = st.t['tgt_rec'].clone()
    fx = (st.res_fx - fx0).cpu().numpy()
    for k, sp in enumerate(st.specs):
        st.check_immunity(DAY, sim=k)
        for key in keys:
            assert torch.equal(got[key][k], st.get(key, k)), (key, k)
        sus = st.get('susceptible', k)
        for v in range(sp.nv):
            want = st.get('rel_sus', k) * (1 - got['sus_imm'][k][v])
            assert torch.equal(rec[v][st.sl(k)][sus].abs(), want[sus])
        at = st.res_slices[k][2] + DAY * L.N_RES_F
        for col, key in ((1, 'sus_imm'), (2, 'symp_imm')):
            assert fx[at + col] == int(torch.round(got[key][k].double() * 2.0 ** L.FX_IMM_BITS).long().sum())
    assert sum(sp.nv == 3 for sp in st.specs) > 1 and st.status() == 0 and keep
    big = int(np.argmax(sizes))
    assert (got['sus_imm'][big] > 0).float().mean() > 0.3
