"""The reference-signature functions called straight into the library against the same
call through the torch operators, and the arguments that must keep going through those."""
import pytest
import torch

import covasim_gb300 as cv
from covasim_gb300 import utils

pytestmark = pytest.mark.gpu


def _args(n=1003, seed=4):
    g = torch.Generator(device='cuda').manual_seed(seed)
    r = lambda: torch.rand(n, generator=g, device='cuda')  # noqa: E731
    b = lambda: r() < 0.5  # noqa: E731
    return dict(load=(85, 60 + 20 * r(), 90 + 9 * r(), torch.full((n,), float('nan'), device='cuda'), 0.3, 2.0, 4.0),
                ts=(r(), r(), b(), b(), 0.6, r(), b(), b(), b(), 0.8, 0.1, 0.2, r()))


def _same(x, y):
    return torch.equal(x.nan_to_num(-7.0), y.nan_to_num(-7.0)) and x.dtype == y.dtype and x.shape == y.shape


@pytest.mark.parametrize('form', ['plain', 'bytes', 'strided', 'double', 'negative view', 'on a stream'])
def test_direct_calls_equal_the_operators(form):
    a = _args()
    load, ts = list(a['load']), list(a['ts'])
    if form == 'bytes':
        ts = [(3 * x.to(torch.uint8)) if torch.is_tensor(x) and x.dtype == torch.bool else x for x in ts]
    elif form == 'strided':
        load[1], ts[0] = load[1].repeat_interleave(2)[::2], ts[0].repeat_interleave(2)[::2]
        ts[2] = ts[2].repeat_interleave(2)[::2]
    elif form == 'double':
        load[1], ts[0] = load[1].double(), ts[0].double()
    elif form == 'negative view':
        load[1], ts[0] = torch._neg_view(-load[1]), torch._neg_view(-ts[0])
    f32 = lambda x: x.clone().to(torch.float32).contiguous()  # noqa: E731
    want_load = torch.ops.covgpu.compute_viral_load(load[0], *(f32(x) for x in load[1:4]), *load[4:])
    u8 = [(x.to(torch.uint8).contiguous() if x.dtype != torch.float64 and not x.is_floating_point() else f32(x))
          if torch.is_tensor(x) else x for x in ts]
    want_ts = torch.ops.covgpu.compute_trans_sus(*u8)
    torch.cuda.synchronize()
    if form == 'on a stream':
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            got_load, got_ts = cv.compute_viral_load(*load), cv.compute_trans_sus(*ts)
        s.synchronize()
    else:
        got_load, got_ts = cv.compute_viral_load(*load), cv.compute_trans_sus(*ts)
    assert _same(got_load, want_load) and all(_same(x, y) for x, y in zip(got_ts, want_ts))


def test_what_torch_may_want_to_see_goes_through_the_operators():
    x = torch.rand(10, device='cuda')
    f = ((torch.float32,),)
    assert utils._direct((x,), f, 5)
    assert not utils._direct((x.cpu(),), f) and not utils._direct((x.double(),), f)
    assert not utils._direct((x.clone().requires_grad_(),), f) and not utils._direct((x[::2],), f)
    assert not utils._direct((x,), f, 1 << 63) and not utils._direct((torch._neg_view(x),), f)
    assert not utils._direct((torch.nn.Parameter(x, requires_grad=False),), f) and not utils._direct((x.cpu().numpy(),), f)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]):
        assert not utils._direct((x,), f)
    with torch.autograd.forward_ad.dual_level():
        assert not utils._direct((x,), f)
    seen = []
    torch.func.vmap(lambda y: seen.append(utils._direct((x,), f)) or y)(x)
    assert seen == [False]
    with torch.utils._python_dispatch.TorchDispatchMode():
        assert not utils._direct((x,), f)
    with pytest.raises((RuntimeError, TypeError, OverflowError)):
        cv.compute_infections(0.1, x.int(), x.int(), x, x, x, seed=1 << 64)
