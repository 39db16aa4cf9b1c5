"""What is timed of covasim_gb300, through its public entry points.

Six kinds of case, each a thing a user of the framework has it do:

* ``viral_load``, ``trans_sus``, ``infections``: the reference-signature functions
  on device tensors, as a day loop of the reference's own would call them once a
  day (and once a layer), at the default 20,000 agents and at millions;
* ``sim``: one simulation run again from day 0 (``Sim.rewind`` and ``Sim.run``), the
  repeated runs of a parameter sweep or an uncertainty study;
* ``fresh``: a simulation made from a population in pinned host memory, run once
  and read back, the first pass of every study;
* ``batch``: many uneven simulations in one ``BatchSim``;
* ``gradient``: a likelihood forward and its backward, the step of a calibration.

The sizes are those of the repository's benchmark, examples and tests: 20,000
agents (the default) to tens of millions, 60 days to a year, random and hybrid
populations, with and without waning immunity, a daily redrawn community layer,
change_beta schedules, testing and tracing, daily importations, and variants.
"""
import math

import numpy as np
import torch

import covasim_gb300 as cv
from covasim_gb300.adjoint import LikelihoodRun

AGENTS_MIN, AGENTS_MAX = 10_000, 20_000_000
AGENT_DAYS_MAX = 800_000_000   # a drawn simulation costs no more than the largest listed one
DAYS_MIN, DAYS_MAX = 40, 365
EDGES_PER_AGENT = 10             # the default random layer: Poisson(20) contacts, 10 undirected edges an agent

SIM = dict(kind='sim', pop_type='hybrid', waning=True, redrawn=True, change_beta=False, testing=False, variants=False,
           imports=0.0)


def listed():
    return [
        # the smallest calls: one day's viral load of the default 20,000-agent sim, where launch latency is all
        dict(name='viral_load_20k', kind='viral_load', agents=20_000),
        # the same step of a million-agent sim (an odd size: populations are not multiples of anything)
        dict(name='trans_sus_1m', kind='trans_sus', agents=1_000_003),
        # one layer of the default sim, and one of a million-agent sim: the reference's compute_infections
        dict(name='infections_20k', kind='infections', agents=20_000, edges=200_000),
        dict(name='infections_1m', kind='infections', agents=1_000_000, edges=9_999_991),
        # the default simulation: 20,000 random agents, 60 days
        dict(SIM, name='sim_default_20k', agents=20_000, days=60, pop_type='random', redrawn=False),
        # a city, with tests, contact tracing and a policy change: the daily work of an outbreak study
        dict(SIM, name='sim_testing_300k', agents=300_000, days=120, testing=True, change_beta=True),
        # the benchmark's headline: a million hybrid agents, 180 days, the community layer redrawn daily
        dict(SIM, name='sim_hybrid_1m', agents=1_000_000, days=180),
        # the largest: a country, three variants, testing and tracing (memory for edges and agents counts)
        dict(SIM, name='sim_variants_10m', agents=10_000_000, days=120, testing=True, variants=True),
        # the first run of a million-agent study, from host memory to results
        dict(SIM, name='fresh_hybrid_1m', kind='fresh', agents=1_000_000, days=180),
        # an ensemble of uneven random sims in one launch sequence
        dict(name='batch_96', kind='batch', sims=96, agents_lo=10_000, agents_hi=500_000, days=120),
        # a calibration step: forward with sensitivities, backward, 100,000 hybrid agents
        dict(name='gradient_100k', kind='gradient', agents=100_000, days=120, every=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['viral_load', 'trans_sus', 'infections', 'sim', 'sim', 'sim', 'fresh', 'batch', 'gradient'])
    if kind in ('viral_load', 'trans_sus'):
        return dict(kind=kind, agents=_log_int(rng, AGENTS_MIN, AGENTS_MAX))
    if kind == 'infections':
        agents = _log_int(rng, AGENTS_MIN, 4_000_000)
        return dict(kind=kind, agents=agents, edges=int(agents * rng.uniform(1.0, 12.0)) | 1)
    if kind == 'batch':
        lo = _log_int(rng, 10_000, 60_000)
        return dict(kind=kind, sims=rng.randint(8, 96), agents_lo=lo, agents_hi=int(lo * rng.uniform(1.5, 8.0)),
                    days=rng.randint(DAYS_MIN, 120))
    days = rng.randint(DAYS_MIN, 200)
    if kind == 'gradient':
        return dict(kind=kind, agents=_log_int(rng, AGENTS_MIN, 200_000), days=min(days, 120),
                    every=rng.choice([5, 10, 20]))
    top = AGENTS_MAX if kind == 'sim' else 2_000_000
    agents = _log_int(rng, AGENTS_MIN, min(top, AGENT_DAYS_MAX // (days + 1)))
    if rng.random() < 0.15:
        days = min(DAYS_MAX, max(days, AGENT_DAYS_MAX // (4 * agents)))
    return dict(SIM, kind=kind, agents=agents, days=days, pop_type=rng.choice(['random', 'hybrid', 'hybrid']),
                waning=rng.random() < 0.8, redrawn=rng.random() < 0.6, change_beta=rng.random() < 0.4,
                testing=rng.random() < 0.4, variants=rng.random() < 0.25, imports=rng.choice([0.0, 0.0, 3.0]))


# ----------------------------------------------------------------------------- the cases' inputs
def _sim(case, seed, gpu_population=True, **kwargs):
    """An uninitialised Sim of the case, its population built on the device."""
    hybrid = case['pop_type'] == 'hybrid'
    pars = dict(pop_size=case['agents'], pop_type=case['pop_type'], n_days=case['days'], rand_seed=seed,
                pop_infected=max(20, case['agents'] // 10_000), use_waning=case['waning'], n_imports=case['imports'])
    if case['redrawn']:
        pars['dynam_layer'] = dict(h=0, s=0, w=0, c=1) if hybrid else dict(a=1)
    interventions = []
    if case['change_beta']:
        interventions.append(cv.change_beta(days=[case['days'] // 3, case['days'] // 2], changes=[0.6, 0.85]))
    if case['testing']:
        interventions += [cv.test_prob(symp_prob=0.1), cv.contact_tracing(trace_probs=0.5)]
    if interventions:
        pars['interventions'] = interventions
    if case['variants']:
        pars['variants'] = [cv.variant(dict(rel_beta=1.5), days=case['days'] // 6, n_imports=100, label='v1.5'),
                            cv.variant(dict(rel_beta=1.7), days=case['days'] // 3, n_imports=100, label='v1.7')]
    return pars, cv.Sim(pars, gpu_population=gpu_population, **kwargs)


def _batch_sizes(case):
    """The uneven population sizes of a batch, log-uniform: the case's, the same for every seed."""
    rng = np.random.default_rng([case['sims'], case['agents_lo'], case['agents_hi']])
    return np.exp(rng.uniform(np.log(case['agents_lo']), np.log(case['agents_hi']), case['sims'])).astype(int).tolist()


def _pinned(x):
    return x.cpu().pin_memory()


def _epidemic(n, gen):
    """A mid-epidemic population's fields, as the reference's day loop has them: 15% infectious, 60% susceptible."""
    u = torch.rand(n, generator=gen, device='cuda')
    nan = torch.full((n,), float('nan'), device='cuda')
    infectious, susceptible = u < 0.15, u >= 0.4
    start = torch.randint(60, 90, (n,), generator=gen, device='cuda').float()
    length = torch.randint(4, 14, (n,), generator=gen, device='cuda').float()
    dead = torch.rand(n, generator=gen, device='cuda') < 0.01
    return dict(infectious=infectious, susceptible=susceptible, u=u,
                start=torch.where(u < 0.4, start, nan),
                recovered=torch.where((u < 0.4) & ~dead, start + length, nan),
                dead=torch.where((u < 0.4) & dead, start + length, nan))


def prepare(case, seed):
    kind = case['kind']
    gen = torch.Generator(device='cuda').manual_seed(seed)
    if kind == 'viral_load':
        e = _epidemic(case['agents'], gen)
        return dict(kind=kind, args=(85, e['start'], e['recovered'], e['dead'], 0.3, 2.0, 4.0))
    if kind == 'trans_sus':
        n = case['agents']
        e = _epidemic(n, gen)
        some = lambda p: torch.rand(n, generator=gen, device='cuda') < p  # noqa: E731
        uniform = lambda: torch.rand(n, generator=gen, device='cuda')  # noqa: E731
        return dict(kind=kind, args=(2 * uniform(), 0.5 + uniform(), e['infectious'], e['susceptible'], 0.6,
                                     0.5 + uniform(), some(0.6), some(0.05), some(0.05), 0.8, 0.1, 0.2,
                                     0.5 * uniform()))
    if kind == 'infections':
        n, m = case['agents'], case['edges']
        e = _epidemic(n, gen)
        p1 = torch.randint(0, n, (m,), generator=gen, device='cuda', dtype=torch.int32).sort().values
        p2 = torch.randint(0, n, (m,), generator=gen, device='cuda', dtype=torch.int32)
        rel_trans = e['infectious'] * (0.5 + torch.rand(n, generator=gen, device='cuda'))
        rel_sus = e['susceptible'] * (0.5 + torch.rand(n, generator=gen, device='cuda'))
        return dict(kind=kind, args=(0.016, p1, p2, torch.ones(m, device='cuda'), rel_trans, rel_sus),
                    options=dict(seed=seed, day=85), room=m // 64)
    if kind == 'sim':
        _, sim = _sim(case, seed)
        sim.initialize()
        return dict(kind=kind, sim=sim, day0=sim.state.snapshot())
    if kind == 'fresh':
        pars, made = _sim(case, seed)
        made.initialize()
        contacts = {k: dict(p1=_pinned(c['p1']), p2=_pinned(c['p2'])) for k, c in made.popdict['contacts'].items()}
        popdict = dict(uid=made.popdict['uid'], age=made.popdict['age'], sex=made.popdict['sex'], contacts=contacts)
        person = {k: _pinned(v) for k, v in made._person.items()}
        return dict(kind=kind, case=case, seed=seed, popdict=popdict, person=person)
    if kind == 'batch':
        rng = np.random.default_rng(seed)
        sims = []
        for k, size in enumerate(_batch_sizes(case)):
            sims.append(cv.Sim(pop_size=size, pop_type='random', contacts=dict(a=int(rng.choice([10, 20, 30]))),
                               beta=float(rng.uniform(0.010, 0.025)), n_days=case['days'], rand_seed=seed + k,
                               interventions=[cv.change_beta(days=30, changes=float(rng.uniform(0.3, 1.0)))],
                               gpu_population=True))
        batch = cv.BatchSim(sims).initialize()
        return dict(kind=kind, batch=batch, day0=batch.state.snapshot())
    if kind == 'gradient':
        sim = cv.Sim(pop_size=case['agents'], pop_type='hybrid', pop_infected=100, n_days=case['days'], rand_seed=seed,
                     dynam_layer=dict(h=0, s=0, w=0, c=1), gpu_population=True,
                     interventions=[cv.change_beta(days=[case['days'] // 4, case['days'] // 2], changes=[0.7, 0.9])])
        run_ = LikelihoodRun(sim, checkpoint_every=case['every'])
        return dict(kind=kind, run=run_, theta=run_.params.theta0 * np.random.default_rng(seed).uniform(0.9, 1.1, len(
            run_.params.theta0)))
    raise ValueError(f'unknown kind {kind}')


# ----------------------------------------------------------------------------- one pass
def _outcome(sim):
    """A finished sim's result series and its agents."""
    g = sim.people.gpu
    return dict(results=np.stack([sim.results[k].values for k in sim.result_keys()]),
                by_variant=np.stack([v.values for v in sim.results['variant'].values()]),
                naive=g('naive'), recovered_variant=g('recovered_variant'), n_infections=g('n_infections'),
                date_exposed=g('date_exposed'), date_recovered=g('date_recovered'), date_dead=g('date_dead'),
                date_end_quarantine=g('date_end_quarantine'), rel_trans=g('rel_trans'), peak_nab=g('peak_nab'),
                nab=g('nab'), sus_imm=g('sus_imm'), symp_imm=g('symp_imm'), sev_imm=g('sev_imm'))


def run(state):
    kind = state['kind']
    if kind == 'viral_load':
        return cv.utils.compute_viral_load(*state['args'])
    if kind == 'trans_sus':
        return cv.utils.compute_trans_sus(*state['args'])
    if kind == 'infections':
        # a day's infections in buffers of a fixed size, as a loop that keeps a log holds them (about 0.3% of the edges)
        return [torch.nn.functional.pad(x, (0, state['room'] - len(x)), value=-1)
                for x in cv.utils.compute_infections(*state['args'], **state['options'])]
    if kind == 'sim':
        sim = state['sim'].rewind(state['day0'])
        return _outcome(sim.run())
    if kind == 'fresh':
        _, sim = _sim(state['case'], state['seed'], gpu_population=False, popdict=state['popdict'],
                      person=state['person'])
        return _outcome(sim.run())
    if kind == 'batch':
        batch = state['batch']
        batch.state.restore(state['day0'])
        batch.run()
        return dict(new_infections=batch.series('new_infections'),
                    agents=[torch.cat([batch.state.get(k, i) for i in range(len(batch.sims))])
                            for k in ('date_exposed', 'date_recovered', 'nab')])
    ll, expected = state['run'].forward(state['theta'])
    return dict(ll=ll, expected=expected, gradient=state['run'].backward(1.0, np.ones(len(expected))),
                **{k: state['run'].last[k] for k in ('G', 'H')})


# ----------------------------------------------------------------------------- its least work
def work(case):
    """Bytes a pass cannot do without. Simulations, per agent and day: the state word, the recovery date and
    rel_sus (12), and with waning the NAb level read and written, its peak and event day (16) and the two daily
    efficacies a variant (8); per stored contact and day one endpoint list (4); the testing dates and state (16)."""
    kind = case['kind']
    if kind == 'viral_load':
        return dict(bytes=16 * case['agents'], flops=0)
    if kind == 'trans_sus':
        return dict(bytes=(4 * 4 + 5 + 2 * 4) * case['agents'], flops=9 * case['agents'])
    if kind == 'infections':
        return dict(bytes=12 * case['edges'] + 8 * case['agents'], flops=0)
    if kind == 'batch':
        return dict(bytes=sum(_batch_sizes(case)) * (case['days'] + 1) * (36 + 4 * EDGES_PER_AGENT), flops=0)
    if kind == 'gradient':
        return dict(bytes=case['agents'] * (case['days'] + 1) * (36 + 4 * 7.75), flops=0)
    variants = 3 if case['variants'] else 1
    agent = 12 + (16 + 8 * variants if case['waning'] else 0) + (16 if case['testing'] else 0)
    if case['pop_type'] == 'hybrid':
        stored = 7.75 + (0 if case['redrawn'] else 10)
    else:
        stored = 0 if case['redrawn'] else EDGES_PER_AGENT
    return dict(bytes=case['agents'] * (case['days'] + 1) * (agent + 4 * stored), flops=0)


# ----------------------------------------------------------------------------- in 64 bits
def exact(case, seed):
    """The two elementwise functions (covasim/utils.py:39-90) in float64; the others return draws' outcomes."""
    if case['kind'] not in ('viral_load', 'trans_sus'):
        return None
    args = [a.to(torch.float64) if torch.is_tensor(a) else a for a in prepare(case, seed)['args']]
    if case['kind'] == 'viral_load':
        t, start, recovered, dead, frac_time, load_ratio, high_cap = args
        total = torch.where(torch.isnan(dead), recovered, dead) - start
        point = torch.where(frac_time * total > high_cap, high_cap / total, torch.full_like(total, frac_time))
        load = torch.where((t - start) / total < point, load_ratio, 1.0)
        return load / (1 + frac_time * (load_ratio - 1))
    (rel_trans, rel_sus, inf, sus, beta_layer, viral_load, symp, iso, quar, asymp_factor, iso_factor, quar_factor,
     immunity) = args
    factor = lambda on, f: torch.where(on.bool(), f, 1.0)  # noqa: E731
    trans = (rel_trans * inf * factor(quar, quar_factor) * factor(~symp.bool(), asymp_factor) *
             factor(iso, iso_factor) * beta_layer * viral_load)
    return trans, rel_sus * sus * factor(quar, quar_factor) * (1 - immunity)
