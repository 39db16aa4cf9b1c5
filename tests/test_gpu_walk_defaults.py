"""The default walk rule's modes that no other test runs, against the streamed pass: a redrawn layer
with testing (one launch a day, behind the test and post passes), batches, and an agent index without
the reverse endpoints (rev1)."""
import numpy as np
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _same(a, b):
    for key in a:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)


@pytest.mark.parametrize('use_graph', [False, True])
@pytest.mark.parametrize('n,days,want', [(2_001, 60, L.WALK_ALL), (20_001, 50, L.WALK_ALL), (200_003, 30, L.WALK_ALL),
                                         (400_003, 25, 32)])
def test_a_redrawn_layer_with_testing(n, days, want, use_graph):
    runs = []
    for asked in (None, 0, -1):
        sim = cv.Sim(dict(pop_type='hybrid', pop_size=n, n_days=days, rand_seed=4, pop_infected=max(20, n // 40),
                          dynam_layer=dict(h=0, s=0, w=0, c=1), interventions=[
                              cv.test_prob(symp_prob=0.1), cv.contact_tracing(trace_probs=0.5)]))
        sim.initialize()
        if asked is None:
            assert sim.state.cstate.src_walk == want
        else:
            sim.state.set_src_walk(asked)
        snap = sim.state.snapshot()
        sim.run(use_graph=use_graph)
        if use_graph:  # the first run of a range is launched directly, the second captured
            sim.rewind(snap).run(use_graph=True)
        st = sim.state
        runs.append((sim.raw_results(), [st.t[k].clone() for k in ('flags', 'dates', 'vstate')], st.infection_log_tensor(0)))
    for other in runs[1:]:
        _same(runs[0][0], other[0])
        assert all(torch.equal(x.view(torch.int32), y.view(torch.int32)) for x, y in zip(runs[0][1], other[1]))
        assert torch.equal(runs[0][2], other[2])
    assert runs[0][0]['new_infections'].sum() > n // 20


@pytest.mark.parametrize('redrawn,testing,sizes,want', [(True, True, (4_001, 900, 31, 20_001), L.WALK_ALL),
                                                        (True, True, (4_001, 380_000), 128),
                                                        (True, False, (4_001, 900, 31), 32),
                                                        (False, False, (1_600_001, 33, 1_500_000), L.WALK_ALL)])
def test_batches(redrawn, testing, sizes, want):
    runs = []
    for asked in (None, 0):
        sims = []
        for k, n in enumerate(sizes):
            pars = dict(pop_type='hybrid' if redrawn else 'random', pop_size=n, rand_seed=k,
                        pop_infected=max(3, n // 30), n_days=25 if max(sizes) < 10**6 else 12)
            if redrawn:
                pars['dynam_layer'] = dict(h=0, s=0, w=0, c=1)
            if testing and k != 1:  # sims with and without a programme
                pars['interventions'] = [cv.test_prob(symp_prob=0.2), cv.contact_tracing(trace_probs=0.5)]
            sims.append(cv.Sim(pars, gpu_population=n > 10**6))
        b = cv.BatchSim(sims).initialize()
        if asked is None:
            assert b.state.cstate.src_walk == want
        else:
            b.state.set_src_walk(asked)
        b.run()
        runs.append([b.results(k) for k in range(len(sizes))])
        del b, sims
    for a, c in zip(*runs):
        _same(a, c)
    assert runs[0][0]['new_infections'].sum() > 0


def test_index_without_the_reverse_endpoints():
    """covgpu_trace_index's index: the walk and the tracing marks read the other endpoint through perm2."""
    runs = []
    for form in ('agent index', 'trace index'):
        sim = cv.Sim(dict(pop_type='hybrid', pop_size=9_001, n_days=50, rand_seed=6, pop_infected=60,
                          interventions=[cv.test_prob(symp_prob=0.4), cv.contact_tracing(trace_probs=0.7)]))
        sim.initialize()
        st = sim.state
        if form == 'trace index':
            keep = []
            for (k, _), seg in st.segment_index.items():
                rec, n = st.segments[seg], st.specs[k].n
                rp = torch.empty((2, n + 1), dtype=torch.int32, device='cuda')
                perm2 = torch.empty(int(rec.n_edges), dtype=torch.int32, device='cuda')
                scratch = torch.empty(int(st.lib.covgpu_trace_index_scratch(n)), dtype=torch.int64, device='cuda')
                L.call('covgpu_trace_index', rec.p1, rec.p2, int(rec.n_edges), int(st.offsets[k]), n, rp[0].data_ptr(),
                       rp[1].data_ptr(), perm2.data_ptr(), scratch.data_ptr(), torch.cuda.current_stream().cuda_stream)
                rec.rp1, rec.rp2, rec.perm2, rec.rev1 = rp[0].data_ptr(), rp[1].data_ptr(), perm2.data_ptr(), None
                keep += [rp, perm2, scratch]
            st._tile_segments()  # the segment table with this index
        st.set_src_walk(-1)
        assert st.cstate.src_walk == L.WALK_ALL and all(bool(r.rev1) == (form == 'agent index') for r in st.segments)
        sim.run(use_graph=False)
        runs.append((sim.raw_results(), sim.state.infection_log_tensor(0)))
    _same(runs[0][0], runs[1][0])
    assert torch.equal(runs[0][1], runs[1][1]) and runs[0][0]['new_quarantined'].sum() > 0
