"""Copies and fills of many arrays in one launch, a run's outcome sums, seed infections of
several sims in one launch, and the draws of variant importations."""
import ctypes as C

import numpy as np
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import _lib as L
from covasim_gb300.sim import mean_infectious_duration

pytestmark = pytest.mark.gpu
STREAM = lambda: C.c_void_p(torch.cuda.current_stream().cuda_stream)  # noqa: E731


@pytest.mark.parametrize('n_spans', [1, 39, 40, 41, 95])
@pytest.mark.parametrize('shift', [0, 1, 4])
def test_copy_spans(n_spans, shift):
    """Sizes around a 16-byte word and a chunk, arrays off a 16-byte boundary, empty spans."""
    rng = np.random.default_rng(n_spans)
    sizes = [0, 1, 15, 16, 17, 8191, 8192, 8193, 100_003]
    spans, checks = [], []
    for k in range(n_spans):
        m = sizes[k % len(sizes)]
        src = torch.from_numpy(rng.integers(0, 256, m + 8, dtype=np.uint8)).cuda()
        dst = torch.full((m + 32,), 7, dtype=torch.uint8, device='cuda')
        fill = (None, 0, 0xFF)[k % 3]
        want = dst.clone()
        want[16 + shift:16 + shift + m] = src[shift:shift + m] if fill is None else fill
        spans.append(L.Span(dst.data_ptr() + 16 + shift, src.data_ptr() + shift if fill is None else None, m,
                            fill or 0, 0))
        checks.append((src, dst, want))
    assert L.lib().covgpu_copy_spans((L.Span * n_spans)(*spans), n_spans, STREAM()) == L.OK
    for _, dst, want in checks:
        assert torch.equal(dst, want)
    assert L.lib().covgpu_copy_spans((L.Span * 1)(L.Span(None, None, 5, 0, 0)), 1, STREAM()) == L.BADARG


@pytest.mark.parametrize('n', [1, 255, 77_825, 300_001])
def test_mean_infectious_duration(n):
    g = torch.Generator(device='cuda').manual_seed(n)
    u = torch.rand(n, generator=g, device='cuda')
    nan = torch.full_like(u, float('nan'))
    inf = torch.where(u < 0.6, (100 * u).round(), nan)
    rec, dead = torch.where(u < 0.5, inf + 9, nan), torch.where((u >= 0.5) & (u < 0.55), inf + 20.5, nan)
    want = mean_infectious_duration(rec.cpu().numpy(), dead.cpu().numpy(), inf.cpu().numpy())
    assert mean_infectious_duration(rec, dead, inf) == want
    assert mean_infectious_duration(nan, nan, nan) == 0.0
    assert mean_infectious_duration(rec.double(), dead.double(), inf.double()) == want


def test_seeds_of_a_batch_in_one_launch_equal_one_by_one():
    make = lambda: cv.BatchSim([cv.Sim(pop_size=n, pop_type='random', n_days=10, rand_seed=n, pop_infected=n // 9,  # noqa: E731
                                       frac_susceptible=f) for n, f in ((33, 1.0), (1000, 0.8), (257, 1.0), (4001, 1.0))])
    a, b = make().initialize(), make().initialize()
    a.seed_infections()
    from covasim_gb300.sim import init_infections
    for k, s in enumerate(b.sims):
        init_infections(b.state, k, s.pars)
    for key in ('flags', 'vstate', 'dates', 'durs', 'peak_nab', 'n_infections'):
        assert torch.equal(a.state.t[key].view(torch.int32), b.state.t[key].view(torch.int32)), key
    for k in range(4):
        assert torch.equal(a.state.infection_log_tensor(k), b.state.infection_log_tensor(k))
    a.run()
    assert np.array_equal(a.series('new_infections'), np.stack([a.results(k)['new_infections'] for k in range(4)]))
    assert np.array_equal(a.series('pop_nabs'), np.stack([a.results(k)['pop_nabs'] for k in range(4)]))
    with pytest.raises(IndexError):
        a.state.infect_sims(0, [(1, [1000])])


def test_choose_susceptible_draws_as_numpy_over_their_indices():
    sim = cv.Sim(pop_size=5003, n_days=30, rand_seed=1, pop_infected=900)
    sim.initialize()
    sim.run(until=12)
    sus = np.nonzero(sim.people['susceptible'])[0]
    for m in (0, 1, 100, len(sus)):
        got = sim.state.choose_susceptible(0, m, np.random.default_rng(m))
        assert np.array_equal(got, np.random.default_rng(m).choice(sus, m, replace=False))
    with pytest.raises(ValueError):
        sim.state.choose_susceptible(0, len(sus) + 1, np.random.default_rng(0))
